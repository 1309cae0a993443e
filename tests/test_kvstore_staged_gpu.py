"""Whole slots beside one another go through the staging buffer, others through the arena's mapping: the same bytes either way."""
import random

import pytest
import torch

from llumnix_kv_b200.kvstore import PinnedKVStore
from llumnix_kv_b200.kvstore import store as S
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LAYERS = 8


def _slots(kind, n, rng):
    if kind == "one run":
        return list(range(3, 3 + n))
    if kind == "two runs":
        return list(range(n // 2, n)) + list(range(n + 5, n + 5 + n // 2))
    return rng.sample(range(2 * n), n)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("kind, staged", [("one run", True), ("two runs", True), ("scattered", False)])
@pytest.mark.parametrize("n", [67, 150])
def test_both_ways_bring_the_same_bytes(ops, fp8, kind, staged, n):
    """67 slots of 512 KiB (264 in fp8): two full halves and a remainder, or one and a remainder."""
    rng = random.Random(n)
    lay = AttnLayout(CacheShape.FLASH, 2 * n + 2, 16, 8, 128, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(LAYERS)]
    stores = [PinnedKVStore("kvx_staged_%d_%d" % (n, i), lay, src, 0, 1, 2 * n + 8, create=True, fp8=fp8) for i in range(2)]
    try:
        stores[1]._staging = None                    # this one goes through the mapping
        blocks, slots = rng.sample(range(2 * n + 2), n), _slots(kind, n, rng)
        big = n * stores[0].slot_bytes >= S._STAGED_LEAST
        assert (stores[0]._runs(slots) is not None) == (staged and big) and stores[1]._runs(slots) is None
        for st in stores:
            st.host.zero_()
        events = [st.save_layers(0, LAYERS, blocks, slots) for st in stores]
        events += [st.save_layers(0, LAYERS, blocks, slots) for st in stores]      # the halves are used again
        for e in events:
            e.synchronize()
        assert torch.equal(stores[0].host, stores[1].host) and bool(stores[0].host.any())
        got = []
        for st in stores:
            for t in src:
                t.zero_()
            torch.cuda.synchronize()
            st.load_layers(0, LAYERS, blocks, slots).synchronize()
            st.check_status()
            got.append([t.clone() for t in src])
        for a, b in zip(*got):
            assert torch.equal(a, b) and bool(a.any())
        # a save that follows a load and overwrites the half it read from, then part of the layers (never staged)
        first, half = [t.clone() for t in src], n // 2
        after = torch.cuda.Event()
        for t in src:
            t.view(torch.int16).bitwise_xor_(0x0101)
        after.record()
        ev = [st.load_layers(0, LAYERS, blocks, slots, after=after) for st in stores]
        ev += [st.save_layers(0, LAYERS, blocks, slots) for st in stores] + [st.save_layers(1, 3, blocks[:half], slots[:half]) for st in stores]
        for e in ev:
            e.synchronize()
        assert torch.equal(stores[0].host, stores[1].host)
        for st in stores:
            st.check_status()
        for t, was in zip(src, first):
            assert torch.equal(lay.view(t, torch.int16)[blocks], lay.view(was, torch.int16)[blocks])
    finally:
        for i, st in enumerate(stores):
            st.close()
            ops.KvStore.unlink("kvx_staged_%d_%d" % (n, i))
