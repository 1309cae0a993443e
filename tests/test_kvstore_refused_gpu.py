"""Block ids outside of the cache: their slots stay as they were and the status says so, whichever way a move would have taken."""
import pytest
import torch

from llumnix_kv_b200.kvstore import PinnedKVStore
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import AttnTransfer, ReqChunk

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LAYERS, N = 8, 70      # slots of 512 KiB: two halves of the buffer and a remainder


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("at", [0, 40, N - 1])
@pytest.mark.parametrize("bad", [N, 2 ** 32 - 1])
def test_a_refused_block_leaves_its_slot_alone(ops, fp8, at, bad):
    lay = AttnLayout(CacheShape.FLASH, N, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(LAYERS)]
    name = "kvx_refused_%d_%d_%d" % (fp8, at, bad)
    st = PinnedKVStore(name, lay, src, 0, 1, N + 4, create=True, fp8=fp8)
    try:
        slots = list(range(2, 2 + N))
        st.save_layers(0, LAYERS, list(range(N)), slots).synchronize()
        want = st.host.view(N + 4, st.slot_bytes).clone()
        assert bool(want[2 + at].any())
        st.host.fill_(0x5A)
        blocks = list(range(N))
        blocks[at] = bad
        st.save_layers(0, LAYERS, blocks, slots).synchronize()
        got = st.host.view(N + 4, st.slot_bytes)
        want[2 + at] = 0x5A
        assert torch.equal(got[2:2 + N], want[2:2 + N]) and bool((got[:2] == 0x5A).all()) and bool((got[2 + N:] == 0x5A).all())
        with pytest.raises(RuntimeError, match="status"):
            st.check_status()
        kept = [t.clone() for t in src]
        st.load_layers(0, LAYERS, blocks, slots).synchronize()
        for t, was in zip(src, kept):      # the block whose id was replaced stays as it was too
            assert torch.equal(lay.view(t, torch.int16)[at], lay.view(was, torch.int16)[at])
    finally:
        st.close()
        ops.KvStore.unlink(name)


def test_one_read_tells_about_all_transfers_of_a_store(ops, monkeypatch):
    lay = AttnLayout(CacheShape.FLASH, N, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(LAYERS)]
    st = PinnedKVStore("kvx_status", lay, src, 0, 1, N, create=True)
    try:
        reads, look = [], AttnTransfer.check_status
        monkeypatch.setattr(AttnTransfer, "check_status", lambda x: reads.append(x) or look(x))
        st.check_status()
        assert len(reads) == 1
        for x in (st._save_xfer, st._load_xfer, st._stage_save, st._stage_load):
            bad, good = [x.src_layout.num_blocks], [0]
            x.launch(x.plan([ReqChunk(bad, good, 0, 16)], stream=st.stream), stream=st.stream)
            st.stream.synchronize()
            with pytest.raises(RuntimeError, match="status"):
                st.check_status()
            x.status.zero_()
            torch.cuda.synchronize()
            st.check_status()
        assert len(reads) == 9
    finally:
        st.close()
        ops.KvStore.unlink("kvx_status")


@pytest.mark.parametrize("fp8", [False, True])
def test_a_first_move_finds_its_plans_memory_at_hand(ops, fp8):
    """A place on the store's stream is there before the first plan asks: getting memory from the driver took up to 10 ms of that move."""
    lay = AttnLayout(CacheShape.FLASH, N, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(LAYERS)]
    st = PinnedKVStore("kvx_first_%d" % fp8, lay, src, 0, 1, N, create=True, fp8=fp8)
    try:
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        events = [f(*at, list(range(n)), list(range(n))) for f in (st.save_layers, st.load_layers) for at in ((0, LAYERS), (1, 2)) for n in (N, 5)]
        assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
        for e in events:
            e.synchronize()
        st.check_status()
    finally:
        st.close()
        ops.KvStore.unlink("kvx_first_%d" % fp8)
