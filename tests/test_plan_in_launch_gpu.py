"""A short plan travels in the launch's parameters: the same bytes as from the device buffer, up to the last plan that fits."""
import random

import pytest
import torch

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import (MODE_BF16_TO_MXFP8, MODE_COPY, MODE_MXFP8_TO_BF16, AttnTransfer, ReqChunk,
                                          reference_transfer)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
L = 2


def _pair(mode, blocks, heads, use_tma):
    src_l = AttnLayout(CacheShape.FLASHINFER, blocks, 16, heads, 64, 1 if mode == MODE_MXFP8_TO_BF16 else 2,
                       mx_scaled=mode == MODE_MXFP8_TO_BF16)
    dst_l = AttnLayout(CacheShape.FLASH if mode != MODE_BF16_TO_MXFP8 else CacheShape.FLASHINFER, blocks, 16, heads, 64,
                       1 if mode == MODE_BF16_TO_MXFP8 else 2, mx_scaled=mode == MODE_BF16_TO_MXFP8)
    src = [src_l.alloc(DEV, "normal", seed=i) if mode != MODE_MXFP8_TO_BF16 else src_l.alloc(DEV) for i in range(L)]
    if mode == MODE_MXFP8_TO_BF16:
        for s in src:
            s.copy_(torch.randint(0, 0x70, s.shape, dtype=torch.uint8, device=DEV))
            sc = src_l.scale_view(s)
            sc.copy_(torch.randint(120, 130, sc.shape, dtype=torch.uint8, device=DEV))
    dst = [dst_l.alloc(DEV) for _ in range(L)]
    x = AttnTransfer(src_l, dst_l, [t.data_ptr() for t in src], [t.data_ptr() for t in dst], DEV, mode=mode, use_tma=use_tma)
    return x, src_l, dst_l, src, dst


def _check(x, src_l, dst_l, src, dst, chunks, mode):
    torch.cuda.synchronize()
    assert x.check_status() == (0, 0)
    for s, d in zip(src, dst):
        want = torch.zeros_like(d)
        reference_transfer(src_l, dst_l, s, want, chunks, None, mode)
        assert torch.equal(d, want)
        d.zero_()


# 32 bytes a request and 4 a block id: (requests, blocks a side of each); 1 x 444 is the last that fits 3584 bytes
@pytest.mark.parametrize("reqs, per_req, fits", [(1, 1, True), (7, 3, True), (1, 444, True), (1, 445, False), (8, 52, True), (8, 53, False)])
@pytest.mark.parametrize("mode, heads, use_tma", [(MODE_COPY, 2, True), (MODE_COPY, 1, False), (MODE_BF16_TO_MXFP8, 2, False),
                                                  (MODE_MXFP8_TO_BF16, 4, False), (MODE_MXFP8_TO_BF16, 1, False)])
def test_same_bytes_from_either_place(ops, mode, heads, use_tma, reqs, per_req, fits):
    blocks = reqs * per_req + 3
    x, src_l, dst_l, src, dst = _pair(mode, blocks, heads, use_tma)
    rng = random.Random(reqs * 1000 + per_req)
    a, b = rng.sample(range(blocks), reqs * per_req), rng.sample(range(blocks), reqs * per_req)
    # a few tokens of every request, beginning and ending inside a block: the oracle goes token by token
    chunks = [ReqChunk(a[i * per_req:(i + 1) * per_req], b[i * per_req:(i + 1) * per_req], max(0, per_req * 16 - 21 - i),
                       min(per_req * 16, 21 + i) - 3) for i in range(reqs)]
    plan = x.plan(chunks)
    assert (plan._dev is None) == fits
    x.launch(plan)
    _check(x, src_l, dst_l, src, dst, chunks, mode)
    assert (plan._dev is None) == fits
    plan.dev                               # from here on its launches read the buffer
    x.launch(plan)
    _check(x, src_l, dst_l, src, dst, chunks, mode)


def test_a_captured_launch_reads_the_buffer(ops):
    x, src_l, dst_l, src, dst = _pair(MODE_COPY, 16, 2, True)
    one, two = [ReqChunk([1, 2], [3, 4], 0, 30)], [ReqChunk([5, 6], [7, 8], 0, 30)]
    s = torch.cuda.Stream()
    plan = x.plan(one)
    x.launch(plan, stream=s)
    s.synchronize()
    assert plan._dev is None
    _check(x, src_l, dst_l, src, dst, one, MODE_COPY)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        x.launch(plan, stream=s)
    g.replay()
    _check(x, src_l, dst_l, src, dst, one, MODE_COPY)
    plan.dev.copy_(x.plan(two).dev)
    g.replay()
    _check(x, src_l, dst_l, src, dst, two, MODE_COPY)
    x.launch(plan)
    _check(x, src_l, dst_l, src, dst, two, MODE_COPY)


@pytest.mark.parametrize("blocks", [444, 445])
def test_a_step_whose_plan_just_fits_and_one_whose_does_not(ops, blocks):
    layers = 5
    lay = AttnLayout(CacheShape.FLASH, 2 * blocks + 2, 16, 2, 64, 2)
    src = [lay.alloc(DEV, "normal", seed=i) for i in range(layers)]
    dst = [lay.alloc(DEV) for _ in range(layers)]
    kw = dict(num_kv_heads=2, cache_shape=int(CacheShape.FLASH))
    srv = KVTransferServer("D|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", dst, [PT.NVLINK], **kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, lay.block_bytes, lay.token_bytes, "fake://", src, [PT.NVLINK], **kw)
    try:
        for step in (1, 2, 3):
            sb, db = list(range(blocks)), list(range(2 * blocks + 1, blocks + 1, -1))
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, blocks * 16, True, sb, db, srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                src[layer].view(torch.int16).add_(1)
                cli.record_event(layer)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for s, d in zip(src, dst):
                assert torch.equal(lay.view(d, torch.int16)[db], lay.view(s, torch.int16)[sb])
    finally:
        cli.drain()
        del cli
        srv.stop()
