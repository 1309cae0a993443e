"""GPU edges of the transfer kernels' data movers: partly filled tiles, head counts and row lengths that are no powers of two,
addresses that are only 16-byte aligned, tiles beyond the range of the fast index division, special values in the quantiser.

Everything here is exact: copies, and codes and scales that the oracle defines bit by bit."""
import random

import pytest
import torch

from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import (MODE_BF16_TO_MXFP8, MODE_COPY, MODE_MXFP8_TO_BF16, AttnTransfer, HeadMap, ReqChunk,
                                          mx_quantize_reference, reference_transfer)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _alloc(lay, seed, shift):
    """A layer whose base is 16 * shift bytes off a 512-byte boundary, filled with normal bf16 values."""
    g = torch.Generator().manual_seed(seed)
    n = lay.layer_bytes
    flat = torch.empty(n + 16 * shift, dtype=torch.uint8, device=DEV)
    view = flat[16 * shift:]
    view.copy_(torch.randn(n // 2 + 1, generator=g).bfloat16().view(torch.uint8)[:n])
    return view


def _chunks(rng, ntpb, edges):
    """One request per (seen, new), with scattered blocks on both sides."""
    need = [-(-(a + b) // ntpb) for a, b in edges]
    pool = sum(need) + 3
    sb, db = rng.sample(range(pool), sum(need)), rng.sample(range(pool), sum(need))
    out, at = [], 0
    for (a, b), n in zip(edges, need):
        out.append(ReqChunk(sb[at:at + n], db[at:at + n], a, b))
        at += n
    return pool, out


def _check(src_l, dst_l, chunks, hm, mode, shift=0, layers=2, prepare=None, **kw):
    src = [_alloc(src_l, 7 + i, shift) for i in range(layers)]
    dst = [_alloc(dst_l, 70 + i, shift) for i in range(layers)]
    if mode == MODE_MXFP8_TO_BF16:
        for s in src:
            src_l.scale_view(s).copy_(torch.randint(100, 150, src_l.scale_view(s).shape, dtype=torch.uint8, device=DEV))
    if prepare is not None:
        for s in src:
            prepare(s)
    want = [d.cpu() for d in dst]
    x = AttnTransfer(src_l, dst_l, [s.data_ptr() for s in src], [d.data_ptr() for d in dst], DEV, head_map=hm, mode=mode, **kw)
    x.launch(x.plan(chunks))
    torch.cuda.synchronize()
    assert x.check_status() == (0, 0)
    for s, d, w in zip(src, dst, want):
        reference_transfer(src_l, dst_l, s.cpu(), w, chunks, hm, mode)
        assert torch.equal(d.cpu(), w)


EDGES = [(0, 1), (0, 15), (0, 16), (0, 17), (15, 1), (15, 2), (3, 9), (16, 31), (1, 46)]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("mode", [MODE_BF16_TO_MXFP8, MODE_MXFP8_TO_BF16])
@pytest.mark.parametrize("heads, dim", [(1, 32), (3, 64), (5, 96), (8, 128), (2, 256)])
def test_quantised_rows_of_any_length_and_alignment(mode, heads, dim, shift):
    pool, chunks = _chunks(random.Random(heads * dim), 16, EDGES)
    wide = AttnLayout(CacheShape.FLASH, pool, 16, heads, dim, 2)
    mx = AttnLayout(CacheShape.FLASHINFER, pool, 16, heads, dim, 1, mx_scaled=True)
    a, b = (wide, mx) if mode == MODE_BF16_TO_MXFP8 else (mx, wide)
    # a NaN code of the random payload has no one bf16 result: the codes are taken without them, as the quantiser writes them
    clean = (lambda s: s.bitwise_and_(0xF7)) if mode == MODE_MXFP8_TO_BF16 else None

    def prep(s):
        clean(s)
        mx.scale_view(s).copy_(torch.randint(100, 150, mx.scale_view(s).shape, dtype=torch.uint8, device=DEV))

    _check(a, b, chunks, HeadMap(0, 0, heads), mode, shift, prepare=prep if clean else None)


def test_quantiser_keeps_zero_groups_and_extremes():
    pool, chunks = _chunks(random.Random(3), 16, [(0, 33)])
    a = AttnLayout(CacheShape.FLASH, pool, 16, 2, 128, 2)
    b = AttnLayout(CacheShape.FLASHINFER, pool, 16, 2, 128, 1, mx_scaled=True)
    big, tiny = 3.3895313892515355e38, 9.183549615799121e-41      # largest and smallest bf16 magnitudes

    def prep(s):
        v = a.view(s, torch.bfloat16)
        v[..., 0:32] = 0.0
        v[..., 32:64] = tiny
        v[..., 64] = -big
        v[..., 65] = big

    _check(a, b, chunks, HeadMap(0, 0, 2), MODE_BF16_TO_MXFP8, prepare=prep)


@pytest.mark.parametrize("dst_remote", [False, True])      # True: the staged form, whose stores this GPU takes as well
@pytest.mark.parametrize("heads", [1, 8])                   # a warp a tile, four warps a tile
def test_quantiser_with_infinities_and_nan(heads, dst_remote):
    """A NaN does not count for its group's scale and keeps a NaN code; a group with an infinity takes the largest scale, 2^127,
    whose reciprocal is zero in the kernel: NaN for the infinity and zero for the rest."""
    pool, chunks = _chunks(random.Random(5), 16, [(0, 37)])
    a = AttnLayout(CacheShape.FLASH, pool, 16, heads, 128, 2)
    b = AttnLayout(CacheShape.FLASHINFER, pool, 16, heads, 128, 1, mx_scaled=True)
    inf, nan = float("inf"), float("nan")
    src, dst = _alloc(a, 1, 0), torch.zeros(b.layer_bytes, dtype=torch.uint8, device=DEV)
    v = a.view(src, torch.bfloat16)
    v[..., 0], v[..., 31] = nan, -nan           # both halves of a group: two lanes of the kernel
    v[..., 32:64] = nan
    v[..., 70] = inf
    v[..., 90], v[..., 91] = nan, -inf
    v[..., 96:128][..., ::2] = nan              # every other value
    x = AttnTransfer(a, b, [src.data_ptr()], [dst.data_ptr()], DEV, head_map=HeadMap(0, 0, heads), mode=MODE_BF16_TO_MXFP8,
                     dst_remote=dst_remote)
    x.launch(x.plan(chunks))
    torch.cuda.synchronize()
    assert x.check_status() == (0, 0)
    f = v.float().cpu()
    q, e = b.view(dst, torch.uint8).cpu(), b.scale_view(dst).cpu()
    c = chunks[0]
    for t in range(37):
        row = f[c.src_blocks[t // 16], :, t % 16]
        want_q, want_e = mx_quantize_reference(torch.where(row.isnan(), torch.zeros(()), row))
        got_q, got_e = q[c.dst_blocks[t // 16], :, t % 16], e[c.dst_blocks[t // 16], :, t % 16]
        assert torch.equal(got_e, want_e)
        is_nan = row.isnan() | row.isinf()
        assert bool(((got_q & 0x7F) == 0x7F)[is_nan].all())
        assert torch.equal(got_q[~is_nan], want_q[~is_nan])


PAIRS = [(CacheShape.FLASH, CacheShape.FLASHINFER), (CacheShape.FLASHINFER, CacheShape.FLASH), (CacheShape.FLASH, CacheShape.FLASH),
         (CacheShape.FLASHINFER, CacheShape.FLASHINFER), (CacheShape.RAGGED_FLASH, CacheShape.FLASHINFER)]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("use_tma", [True, False])
@pytest.mark.parametrize("heads, hm", [(4, HeadMap(0, 0, 4)), (5, HeadMap(2, 1, 3)), (2, HeadMap(1, 0, 1))])
@pytest.mark.parametrize("shapes", PAIRS)
def test_partly_filled_tiles(shapes, heads, hm, use_tma, shift):
    pool, chunks = _chunks(random.Random(heads), 16, EDGES)
    a, b = (AttnLayout(s, pool, 16, heads, 128, 2) for s in shapes)
    _check(a, b, chunks, hm, MODE_COPY, shift, use_tma=use_tma)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("stages", [1, 2, 5])
def test_partly_filled_tiles_in_both_tile_orders_and_any_depth(order, stages):
    pool, chunks = _chunks(random.Random(order), 16, EDGES * 3)
    a, b = (AttnLayout(s, pool, 16, 2, 128, 2) for s in (CacheShape.FLASH, CacheShape.FLASHINFER))
    _check(a, b, chunks, HeadMap(0, 0, 2), MODE_COPY, tile_order=order, store_form=0, tma_stages=stages)


def test_tile_beyond_the_range_of_the_multiplied_division():
    """256 tokens x 33 heads x 16 words = 135168 chunks of a tile, and a ragged one of 251 tokens."""
    pool, chunks = _chunks(random.Random(9), 256, [(0, 256), (2, 251)])
    a, b = (AttnLayout(s, pool, 256, 33, 128, 2) for s in (CacheShape.FLASH, CacheShape.FLASHINFER))
    _check(a, b, chunks, HeadMap(0, 0, 33), MODE_COPY, layers=1, use_tma=False)


@pytest.mark.parametrize("mode", [MODE_BF16_TO_MXFP8, MODE_MXFP8_TO_BF16])
@pytest.mark.parametrize("simt_tile", [0, 1, 2, 4])
@pytest.mark.parametrize("heads, hm, tile_tokens, dst", [
    (4, HeadMap(1, 2, 2), 16, CacheShape.FLASHINFER),     # a window of the heads: one run per head or token
    (1, HeadMap(0, 0, 1), 1, CacheShape.FLASHINFER),      # single rows, scale runs of 4 bytes: read where they are
    (3, HeadMap(0, 0, 3), 4, CacheShape.QWEN3_NEXT_FLASH),
    (4, HeadMap(0, 0, 4), 16, CacheShape.QWEN3_NEXT_FLASH),   # scale bytes of a head apart: read where they are
    (16, HeadMap(0, 0, 16), 4, CacheShape.FLASHINFER),    # a run of four rows and one of 16 scale bytes per head
    (40, HeadMap(0, 0, 40), 16, CacheShape.FLASHINFER),   # tiles larger than a stage of the expansion kernel
])
def test_every_way_of_reading_a_tile_gives_the_same_bytes(heads, hm, tile_tokens, dst, simt_tile, mode):
    pool, chunks = _chunks(random.Random(heads), 16, EDGES)
    wide = AttnLayout(CacheShape.FLASH, pool, 16, heads, 128, 2)
    mx = AttnLayout(dst, pool, 16, heads, 128, 1, mx_scaled=True)
    a, b = (wide, mx) if mode == MODE_BF16_TO_MXFP8 else (mx, wide)

    def prep(s):
        s.bitwise_and_(0xF7)
        mx.scale_view(s).copy_(torch.randint(100, 150, mx.scale_view(s).shape, dtype=torch.uint8, device=DEV))

    _check(a, b, chunks, hm, mode, layers=1, prepare=prep if mode == MODE_MXFP8_TO_BF16 else None, tile_tokens=tile_tokens,
           simt_tile=simt_tile)


@pytest.mark.parametrize("mode", [MODE_COPY, MODE_MXFP8_TO_BF16])
def test_more_tiles_than_the_grid_and_a_padded_tail(mode):
    """A launch whose CTAs pass several tiles through their stages, with tail slots to zero behind a partly filled tile."""
    pool, chunks = _chunks(random.Random(4), 16, [(5, 3000), (0, 4001), (16, 777)])
    for c in chunks:
        c.pad_tail = True
    wide = AttnLayout(CacheShape.FLASH, pool, 16, 2, 128, 2)
    mx = AttnLayout(CacheShape.FLASHINFER, pool, 16, 2, 128, 1, mx_scaled=True)
    hnd = AttnLayout(CacheShape.FLASHINFER, pool, 16, 2, 128, 2)

    def prep(s):
        s.bitwise_and_(0xF7)
        mx.scale_view(s).copy_(torch.randint(100, 150, mx.scale_view(s).shape, dtype=torch.uint8, device=DEV))

    if mode == MODE_COPY:
        _check(wide, hnd, chunks, HeadMap(0, 0, 2), mode, layers=3)
    else:
        _check(mx, wide, chunks, HeadMap(0, 0, 2), mode, layers=3, prepare=prep)
