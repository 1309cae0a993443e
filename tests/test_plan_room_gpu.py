"""A plan's device buffer beside the allocator's other users: temporaries of a capture, and blocks whose last kernels are pending."""
import pytest
import torch

from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import AttnTransfer, PlanRoom, ReqChunk, reference_transfer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CHUNKS = [ReqChunk([1, 2], [3, 4], 0, 30), ReqChunk([5], [6], 3, 9)]


def _pair():
    src_l, dst_l = (AttnLayout(s, 16, 16, 2, 64, 2) for s in (CacheShape.FLASH, CacheShape.FLASHINFER))
    src, dst = src_l.alloc(DEV, "normal", seed=1), dst_l.alloc(DEV)
    return AttnTransfer(src_l, dst_l, [src.data_ptr()], [dst.data_ptr()], DEV), src_l, dst_l, src, dst


@pytest.mark.parametrize("made", ["before", "on the captured stream", "in the capture"])
def test_a_capture_with_temporaries_of_the_plans_size(ops, made):
    """Zeros are what a replay would write over a plan that shared a temporary's block: no descriptor would point anywhere."""
    x, src_l, dst_l, src, dst = _pair()
    s = torch.cuda.Stream()
    x.launch(x.plan(CHUNKS), stream=s)                    # modules are loaded outside of the capture
    plan = None if made == "in the capture" else x.plan(CHUNKS, stream=s if made == "on the captured stream" else None)
    torch.cuda.synchronize()
    g, temporaries = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(g, stream=s):
        for n in (16, 512, 1024, 4096, PlanRoom.PLACES * ops.KVT_PLAN_IN_LAUNCH):
            t = torch.empty(n, dtype=torch.uint8, device=DEV)
            t.zero_()
            temporaries.append((t.data_ptr(), t.data_ptr() + n))
            del t
        if plan is None:
            plan = x.plan(CHUNKS)
        x.launch(plan, stream=s)
    if made != "in the capture":                          # there the graph fills the buffer itself, behind the temporaries
        assert all(plan.reqs_ptr + plan.nbytes <= a or plan.reqs_ptr >= b for a, b in temporaries)
    want = torch.zeros_like(dst)
    reference_transfer(src_l, dst_l, src, want, CHUNKS)
    for _ in range(3):
        dst.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(dst, want) and x.check_status() == (0, 0)
    assert bytes(plan.dev.cpu().numpy()) == plan._host.blob


@pytest.mark.parametrize("stream", ["current", "another"])
def test_a_buffer_whose_block_is_still_being_written(ops, stream):
    x, src_l, dst_l, src, dst = _pair()
    want = torch.zeros_like(dst)
    reference_transfer(src_l, dst_l, src, want, CHUNKS)
    s = torch.cuda.current_stream() if stream == "current" else torch.cuda.Stream()
    x.launch(x.plan(CHUNKS), stream=s)
    big = torch.empty(1 << 30, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    dst.zero_()
    torch.cuda.synchronize()
    x._room = PlanRoom(x.device, ops.KVT_PLAN_IN_LAUNCH)                          # the next plan takes a slab
    with torch.cuda.stream(s):
        for _ in range(8):
            big.fill_(1)                                  # keeps the stream busy for about a millisecond
        blocks = [torch.empty(PlanRoom.PLACES * ops.KVT_PLAN_IN_LAUNCH, dtype=torch.uint8, device=DEV) for _ in range(4)]
        for b in blocks:
            b.zero_()
        freed = {b.data_ptr() for b in blocks}
        del blocks, b
    plan = x.plan(CHUNKS, stream=None if stream == "current" else s)
    assert plan._place[0].memory.data_ptr() in freed      # or this shows nothing
    plan.dev
    x.launch(plan, stream=s)
    torch.cuda.synchronize()
    assert bytes(plan.dev.cpu().numpy()) == plan._host.blob
    assert torch.equal(dst, want) and x.check_status() == (0, 0)
