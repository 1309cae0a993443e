"""Where a plan's device buffer comes from: it is there before a launch, or a capture, asks for it."""
import threading
import types

import pytest
import torch

from llumnix_kv_b200.ops import p2d_attn
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import AttnTransfer, ReqChunk

CHUNKS = [ReqChunk([1, 2], [3, 4], 0, 30), ReqChunk([5], [6], 3, 9)]


def _no_allocation(monkeypatch):
    def refuse(*a, **kw):
        raise AssertionError("allocated when the buffer was asked for")

    for name in ("empty", "zeros", "empty_like", "tensor"):
        monkeypatch.setattr(torch, name, refuse)


def test_asking_for_the_buffer_allocates_nothing(ops, monkeypatch):
    lay = AttnLayout(CacheShape.FLASH, 8, 16, 2, 64, 2)
    src, dst = lay.alloc("cpu"), lay.alloc("cpu")
    x = AttnTransfer(lay, lay, [src.data_ptr()], [dst.data_ptr()], "cpu", use_tma=False)
    plan = x.plan(CHUNKS)
    _no_allocation(monkeypatch)
    assert bytes(plan.dev.numpy()) == plan._host.blob and plan.block_ids_ptr == plan.reqs_ptr + plan.pool_offset


@pytest.fixture
def fake_cuda(monkeypatch):
    """Streams of a device that is not there: `now` is the current one, `capturing` those in a capture, slabs are CPU tensors."""
    st = types.SimpleNamespace(now=7, capturing=set(), entered=[], recorded=[])
    events = iter(range(1000, 2000))

    class Event:
        def __init__(self):
            self.cuda_event = next(events)

        def record(self, stream):
            st.recorded.append((self.cuda_event, stream.cuda_stream))

    class Entered:
        def __init__(self, stream):
            self.stream = stream

        def __enter__(self):
            st.entered.append(self.stream.cuda_stream)

        def __exit__(self, *a):
            st.entered.pop()

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: types.SimpleNamespace(cuda_stream=st.now))
    monkeypatch.setattr(torch.cuda, "stream", Entered)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: st.entered[-1] in st.capturing)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: st.now, raising=False)
    return st


def test_places_are_apart_and_of_their_streams(fake_cuda):
    room = p2d_attn.PlanRoom(torch.device("cpu"), 3584)
    taken = []
    for i in range(5 * room.PLACES):
        fake_cuda.now = 7 + i % 3
        slab, at = room.take()
        assert 0 <= at and at + 3584 <= slab.memory.numel() and at % 128 == 0
        assert fake_cuda.recorded.count((slab.ready.cuda_event, fake_cuda.now)) == 1
        taken.append((slab, at))
    assert len({(id(slab), at) for slab, at in taken}) == len(taken)
    for s in range(100, 100 + 3 * room.STREAMS):
        room.take(types.SimpleNamespace(cuda_stream=s))
    assert len(room._slabs) == room.STREAMS


def test_threads_take_different_places(fake_cuda):
    room, taken = p2d_attn.PlanRoom(torch.device("cpu"), 3584), []

    def some():
        for _ in range(500):
            taken.append(room.take(types.SimpleNamespace(cuda_stream=3)))

    threads = [threading.Thread(target=some) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len({(id(slab), at) for slab, at in taken}) == len(taken) == 2000


def test_in_a_capture_no_slab_is_made(fake_cuda, ops, monkeypatch):
    room = p2d_attn.PlanRoom(torch.device("cpu"), 3584)
    fake_cuda.capturing.add(7)
    assert room.take() is None and not room._slabs
    fake_cuda.capturing.clear()
    plans = [p2d_attn.DevicePlan(CHUNKS, 16, 16, "cpu", room=room) for _ in range(2)]
    fake_cuda.capturing.add(7)
    _no_allocation(monkeypatch)
    copies = []
    for p in plans:
        p._host = types.SimpleNamespace(copy_to_device=lambda dst, after: copies.append((dst, after)))
        assert p._dev is None and p.dev is p.dev and p.dev.numel() == p.nbytes
    # each filled once, behind the event that says that the memory is free, at a place of its own
    (a, ready), (b, same) = copies
    assert b - a >= plans[0].nbytes and ready == same == fake_cuda.recorded[0][0]
    slab, _ = plans[0]._place
    assert slab.memory.data_ptr() <= a and b + plans[1].nbytes <= slab.memory.data_ptr() + slab.memory.numel()
