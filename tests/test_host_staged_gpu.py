"""The shared-memory transport between GPU caches: gathers run ahead of the frames, and a frame's blob crosses PCIe as one copy into
a staging buffer where it is long enough."""
import time

import pytest
import torch

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# bytes of a layer's frame: 64 KiB (read through the mapping), 512 KiB less and plus a block (either side of the staging rule),
# 2.5 MiB (more layers than the ring holds), 144 and 146 scattered runs (the first list that does not travel in a launch), 17 MiB,
# 33 MiB (more than is staged)
@pytest.mark.parametrize("blocks, layers", [(1, 3), (7, 12), (8, 12), (40, 11), (72, 4), (73, 4), (272, 6), (529, 3)])
@pytest.mark.parametrize("scattered", [True, False])
@pytest.mark.parametrize("gap_s", [0.0, 0.002])
def test_every_layer_arrives(ops, blocks, layers, scattered, gap_s):
    lay = AttnLayout(CacheShape.FLASH, 2 * blocks + 4, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(layers)]
    dst = [lay.alloc(DEV) for _ in range(layers)]
    kw = dict(num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [PT.SHM], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.SHM], **kw)
    try:
        for step in (1, 2):
            sb = list(range(1, blocks + 1))
            db = list(range(2 * blocks + 2, blocks + 2, -1)) if scattered else list(range(blocks + 2, 2 * blocks + 2))
            tokens = blocks * 16 - 5 * step
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, tokens, True, sb, db, srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                src[layer].view(torch.int16).add_(layer + step)
                cli.record_event(layer)
                time.sleep(gap_s)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            for s, d in zip(src, dst):
                want, got = lay.view(s, torch.int16)[sb].movedim(1, 2), lay.view(d, torch.int16)
                assert torch.equal(got[db].movedim(1, 2).reshape(-1, 2, 8, 128)[:tokens], want.reshape(-1, 2, 8, 128)[:tokens])
                rest = torch.ones(lay.num_blocks, dtype=torch.bool, device=DEV)
                rest[db] = False
                assert not bool(got[rest].any())
    finally:
        cli.drain()
        del cli
        srv.stop()


def test_two_tensors_a_layer_and_a_following_smaller_step(ops):
    """An MLA cache's two lists are kept beside one another; the next step's are others."""
    layers, toks, block, n = 9, [132, 656], 64, 70
    src = [[torch.randint(0, 256, (n * block * t,), dtype=torch.uint8, device=DEV) for t in toks] for _ in range(layers)]
    dst = [[torch.zeros(n * block * t, dtype=torch.uint8, device=DEV) for t in toks] for _ in range(layers)]
    kw = dict(num_kv_heads=1, cache_shape=int(CacheShape.DPSK_V32_SPARSE_MLA))
    sizes = [block * t for t in toks]
    srv = KVTransferServer("D|0|1", 1, 0, 0, sizes, toks, "fake://", dst, [PT.SHM], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, sizes, toks, "fake://", src, [PT.SHM], **kw)
    try:
        for step, (sb, db) in enumerate([(list(range(1, 33)), list(range(66, 34, -1))), ([40], [3]), ([50, 52], [5, 9])], 1):
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, len(sb) * block, True, sb, db, srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                cli.record_event(layer)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            for s, d in zip(src, dst):
                for a, b, size in zip(s, d, sizes):
                    assert torch.equal(b.view(n, size)[db], a.view(n, size)[sb])
    finally:
        cli.drain()
        del cli
        srv.stop()


def test_steps_of_other_lengths_share_the_ring(ops):
    """The segment's slots have a step's own length: whatever the step before left, no layer is gathered over one that is still read."""
    layers, most = 23, 130
    lay = AttnLayout(CacheShape.FLASH, 2 * most + 2, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(layers)]
    dst = [lay.alloc(DEV) for _ in range(layers)]
    kw = dict(num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [PT.SHM], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.SHM], **kw)
    try:
        for step, n in enumerate((most, 97, 53, 129, 41, 128, 100), 1):
            sb, db = list(range(n)), list(range(2 * most, 2 * most - 2 * n, -2))
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, n * 16, True, sb, db, srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                src[layer].view(torch.int16).add_(layer + step)
                cli.record_event(layer)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            for s, d in zip(src, dst):
                assert torch.equal(lay.view(d, torch.int16)[db], lay.view(s, torch.int16)[sb])
    finally:
        cli.drain()
        del cli
        srv.stop()
