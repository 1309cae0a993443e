"""Layer events: plain ones inside the process, interprocess ones from when a peer has asked for them."""
import pytest
import torch

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("asked_at", [0, 3, 6])
def test_peer_events_stand_for_every_layer(ops, asked_at):
    """Asked for before, amid and after the layers of a step: a stream that waits for a layer's peer event sees what the forward
    stream wrote before it recorded that layer, in that step and in the next ones."""
    layers = 6
    lay = AttnLayout(CacheShape.FLASH, 8, 16, 8, 128, 2)
    src, dst = [lay.alloc(DEV) for _ in range(layers)], [lay.alloc(DEV) for _ in range(layers)]
    kw = dict(num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [PT.NVLINK], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.NVLINK], **kw)
    try:
        fwd, peer = torch.cuda.Stream(), torch.cuda.Stream()
        big = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
        seen = [torch.zeros_like(t) for t in src]
        torch.cuda.synchronize()
        for step in (1, 2, 3):
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, 64, True, [1, 2, 3, 4], [4, 3, 2, 1], srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                if layer == asked_at:
                    cli._c.share_layer_events()
                with torch.cuda.stream(fwd):
                    big.fill_(layer)                     # the layer is produced "late"
                    src[layer].fill_(10 * step + layer)
                    cli.record_event(layer, fwd)
            cli.flush_send_step()
            cli._c.share_layer_events()
            for layer in range(layers):
                peer.wait_event(cli._peer_events[layer])
                with torch.cuda.stream(peer):
                    seen[layer].copy_(src[layer], non_blocking=True)
            peer.synchronize()
            for layer in range(layers):
                assert int(seen[layer].min()) == int(seen[layer].max()) == 10 * step + layer
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                got = lay.view(dst[layer].view(torch.uint8), torch.int16)[[1, 2, 3, 4]]
                v = 10 * step + layer
                assert bool((got == v * 257).all())
    finally:
        cli.drain()
        del cli
        srv.stop()


def test_a_host_driven_transport_follows_the_layers_after_they_were_shared(ops):
    """Shared-memory frames beside a peer that has asked for the events: no layer leaves before the forward pass has written it."""
    layers = 6
    lay = AttnLayout(CacheShape.FLASH, 8, 16, 8, 128, 2)
    src, dst = [lay.alloc(DEV) for _ in range(layers)], [lay.alloc(DEV) for _ in range(layers)]
    kw = dict(num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [PT.SHM], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.SHM], **kw)
    try:
        fwd = torch.cuda.Stream()
        big = torch.empty(1 << 30, dtype=torch.uint8, device=DEV)
        torch.cuda.synchronize()
        for step in (1, 2, 3):
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, 64, True, [1, 2, 3, 4], [4, 3, 2, 1], srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                with torch.cuda.stream(fwd):
                    for _ in range(8):
                        big.fill_(layer)                 # the layer is produced "late"
                    src[layer].fill_(10 * step + layer)
                    cli.record_event(layer, fwd)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            for layer in range(layers):
                got = lay.view(dst[layer].view(torch.uint8), torch.int16)[[1, 2, 3, 4]]
                assert bool((got == (10 * step + layer) * 257).all())
            cli._c.share_layer_events()
    finally:
        cli.drain()
        del cli
        srv.stop()
