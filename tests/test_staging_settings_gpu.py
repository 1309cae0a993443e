"""How much GPU memory staging takes, and that everything arrives without it."""
import pytest
import torch

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer
from llumnix_kv_b200.kvstore import PinnedKVStore
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(ops, proto):
    """A step of three layers of 16 MiB; the GPU memory that was taken meanwhile."""
    lay = AttnLayout(CacheShape.FLASH, 520, 16, 8, 128, 2)
    src, dst = [lay.alloc(DEV, "normal", seed=i) for i in range(3)], [lay.alloc(DEV) for _ in range(3)]
    kw = dict(num_kv_heads=8, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [proto], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [proto], **kw)
    try:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        blocks = list(range(3, 3 + 256))
        cli.submit_req_send2("D|0|1", 0, "r", 0, 256 * 16, True, blocks, blocks[::-1], srv.worker_info(), stepid=1)
        cli.start_send_step(1, 1)
        for layer in range(3):
            cli.record_event(layer)
        cli.flush_send_step()
        assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
        taken = before - torch.cuda.mem_get_info()[0]
        for s, d in zip(src, dst):
            assert torch.equal(lay.view(s, torch.int16)[blocks], lay.view(d, torch.int16)[blocks[::-1]])
        return taken
    finally:
        cli.drain()
        del cli
        srv.stop()


@pytest.mark.parametrize("proto", [PT.SHM, PT.TCP])
def test_frames_take_what_the_setting_allows(ops, monkeypatch, proto):
    taken = {}
    try:
        for mib in ("4", "0", "-1", "32"):      # frames are longer than 4 MiB: nothing is staged then
            monkeypatch.setenv("BLLM_KVTRANS_STAGING_MB", mib)
            ops.envcfg_reset_for_test()
            taken[mib] = _step(ops, proto)
    finally:
        monkeypatch.delenv("BLLM_KVTRANS_STAGING_MB")
        ops.envcfg_reset_for_test()
    # the frame of 16 MiB is all that differs; 2 MiB is what the driver hands out at a time
    assert taken["32"] - taken["0"] >= 14 << 20 and abs(taken["-1"] - taken["0"]) <= 4 << 20 and taken["4"] - taken["0"] <= 6 << 20


def test_a_store_without_the_buffer(ops, monkeypatch):
    lay = AttnLayout(CacheShape.FLASH, 70, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(8)]
    was = [t.clone() for t in src]
    monkeypatch.setenv("BLLM_KVSTORE_STAGING", "0")
    st = PinnedKVStore("kvx_unstaged", lay, src, 0, 1, 70, create=True)
    try:
        assert st._staging is None
        order = list(range(70))
        st.save_layers(0, 8, order, order).synchronize()
        for t in src:
            t.zero_()
        torch.cuda.synchronize()
        st.load_layers(0, 8, order, order).synchronize()
        st.check_status()
        assert all(torch.equal(t, w) for t, w in zip(src, was))
    finally:
        st.close()
        ops.KvStore.unlink("kvx_unstaged")
