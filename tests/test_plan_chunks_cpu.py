"""Chunk objects that are no plain lists of plain ints: packed, or refused, as their tuples are."""
import decimal

import numpy as np
import pytest
import torch

from llumnix_kv_b200.ops.p2d_attn import DevicePlan, ReqChunk


class Index:
    def __index__(self):
        return 2


class Raises:
    def __index__(self):
        raise RuntimeError("no")


NUMBERS = {"np.float32": np.float32(2), "a fraction": np.float32(1.5), "np.float64": np.float64(2), "float": 2.0, "decimal": decimal.Decimal(2),
           "torch": torch.tensor(2.0), "index": Index(), "raises": Raises(), "bool": True, "largest": 2 ** 32 - 1, "beyond": 2 ** 32,
           "np beyond": np.int64(2 ** 32), "far beyond": 2 ** 70, "below": -1, "np below": np.int8(-1), "text": "2", "none": None}


def _outcome(pack):
    try:
        return pack()
    except Exception as e:
        return type(e)


@pytest.mark.parametrize("what", sorted(NUMBERS))
def test_numbers_convert_as_in_tuples(ops, what):
    v = NUMBERS[what]
    for chunk in (ReqChunk([1, v], [3, 4], 0, 30), ReqChunk([1, 2], [v, 4], 0, 30), ReqChunk([1], [3], v, 9), ReqChunk([1], [3], 0, v)):
        want = _outcome(lambda: ops.kvt_pack_plan([chunk.as_tuple()], 16, 16)[0])
        assert _outcome(lambda: ops.kvt_pack_chunks([chunk], 16, 16).blob) == want


class Shifted(ReqChunk):
    """Says something else in its tuple than in its fields."""
    def as_tuple(self):
        src, dst, seen, new, flags = super().as_tuple()
        return [b + 1 for b in src], dst, seen, new, flags


class Bare:
    """No chunk, but it has a chunk's tuple."""
    def as_tuple(self):
        return [5], [6], 0, 16, 1


class Wrong(Bare):
    def as_tuple(self):
        return [5], [6], 0, -16, 1


def test_a_class_with_a_tuple_of_its_own_is_heard(ops):
    chunks = [ReqChunk([1, 2], [3, 4], 0, 30), Shifted([1, 2], [3, 4], 0, 30), Bare()]
    plan = DevicePlan(chunks, 16, 16, "cpu")
    want = ops.kvt_pack_plan([c.as_tuple() for c in chunks], 16, 16)
    assert (plan._host.blob, plan.n_reqs, plan.total_tiles, plan.pool_offset) == want
    for bad in (Wrong(), object(), None):
        with pytest.raises((TypeError, AttributeError)):
            DevicePlan([bad], 16, 16, "cpu")
