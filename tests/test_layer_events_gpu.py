"""What the client says about its layer events, before and after a peer has asked for them."""
import logging

import pytest
import torch

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LAYERS = 4


@pytest.fixture
def pair(ops):
    lay = AttnLayout(CacheShape.FLASH, 8, 16, 8, 128, 2)
    src, dst = [lay.alloc(DEV) for _ in range(LAYERS)], [lay.alloc(DEV) for _ in range(LAYERS)]
    kw = dict(num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [PT.NVLINK], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.NVLINK], **kw)
    yield srv, cli
    cli.drain()
    del cli
    srv.stop()


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("late", [False, True])
def test_a_flush_ahead_of_the_last_layer_is_noted(pair, caplog, shared, late):
    srv, cli = pair
    big = torch.empty(1 << 30, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    if shared:
        cli._c.share_layer_events()
    cli.submit_req_send2("D|0|1", 0, "r", 0, 64, True, [1, 2, 3, 4], [4, 3, 2, 1], srv.worker_info(), stepid=1)
    cli.start_send_step(1, 1)
    if late:
        for _ in range(100):
            big.fill_(1)                # tens of milliseconds
    for layer in range(LAYERS):
        cli.record_event(layer)
    if not late:
        torch.cuda.synchronize()
    with caplog.at_level(logging.INFO, logger="llumnix_kv_b200"):
        cli.flush_send_step()
    assert any("before the last layer event" in r.message for r in caplog.records) == late
    assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()


def test_interprocess_events_are_made_when_a_peer_asks(ops, monkeypatch):
    real, made = torch.cuda.Event, []

    def event(*a, **kw):
        made.append(bool(kw.get("interprocess", False)))
        return real(*a, **kw)

    monkeypatch.setattr(torch.cuda, "Event", event)
    lay = AttnLayout(CacheShape.FLASH, 8, 16, 8, 128, 2)
    src = [lay.alloc(DEV) for _ in range(LAYERS)]
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.NVLINK],
                           num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    try:
        assert made == [False] * LAYERS
        s, seen, big = torch.cuda.Stream(), torch.zeros_like(src[0]), torch.empty(1 << 30, dtype=torch.uint8, device=DEV)
        torch.cuda.synchronize()
        for v in (1, 2, 3):
            for _ in range(20):
                big.fill_(v)
            src[-1].fill_(v)
            cli._c.record_layer_event(cli._event_addrs[-1], torch.cuda.current_stream().cuda_stream)
            if v == 2:
                cli._c.share_layer_events()     # carries over what is pending
            s.wait_event(cli._peer_events[-1])
            with torch.cuda.stream(s):
                seen.copy_(src[-1], non_blocking=True)
            s.synchronize()
            assert int(seen.min()) == int(seen.max()) == v
            assert cli._c.layer_event_ready(LAYERS - 1)
    finally:
        cli.drain()
        del cli
