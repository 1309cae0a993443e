"""Packing a plan from chunk objects: the same bytes as from tuples, whatever the ids come in, and the same refusals."""
import random

import numpy as np
import pytest
import torch

from llumnix_kv_b200.ops.p2d_attn import ReqChunk

AS = {"list": list, "tuple": tuple, "numpy": lambda v: np.array(v, dtype=np.int64), "torch": torch.tensor, "iterator": iter,
      "bool": lambda v: [bool(x & 1) for x in v]}


@pytest.mark.parametrize("form", sorted(AS))
@pytest.mark.parametrize("tile, ntpb", [(16, 16), (1, 16), (16, 64)])
def test_chunks_pack_as_tuples_do(ops, form, tile, ntpb):
    rng = random.Random(tile * 131 + ntpb)
    for n in (0, 1, 7):
        def chunks():
            r = random.Random(n)
            return [ReqChunk(AS[form]([r.randrange(2 ** 31) for _ in range(r.randrange(9))]), AS[form]([r.randrange(99) for _ in range(3)]),
                             r.choice([0, 5, 5.0, np.int32(7)]), r.choice([0, 1, 40]), r.random() < 0.5) for _ in range(n)]
        want = ops.kvt_pack_plan([c.as_tuple() for c in chunks()], tile, ntpb)
        got = ops.kvt_pack_chunks(chunks() if rng.random() < 0.5 else iter(chunks()), tile, ntpb)
        assert (got.blob, got.n_reqs, got.total_tiles, got.pool_offset) == want and got.nbytes == len(want[0])


@pytest.mark.parametrize("ids", [[1.5], [-1], [2 ** 32], ["1"], [None], None, 3])
def test_what_is_no_block_id_is_refused(ops, ids):
    for chunk in (ReqChunk(ids, [1], 0, 16), ReqChunk([1], ids, 0, 16)):
        with pytest.raises((TypeError, ValueError, OverflowError)):
            ops.kvt_pack_plan([chunk.as_tuple()], 16, 16)
        with pytest.raises((TypeError, ValueError, OverflowError)):
            ops.kvt_pack_chunks([chunk], 16, 16)
