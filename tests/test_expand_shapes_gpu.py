"""fp8 -> bf16 by the bulk-fed kernel at the edges of its launch shapes: small and large tiles, stages that just fit and that do not."""
import pytest
import torch

from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import MODE_MXFP8_TO_BF16, AttnTransfer, ReqChunk, reference_transfer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# bytes of codes a tile: 4 KiB (the least), 6 KiB (small), 15.5 KiB of 32-byte rows, 8 KiB (the least large), 32, 48 KiB (one stage),
# 50 KiB (no stage: the SIMT kernel serves it)
@pytest.mark.parametrize("heads, dim", [(2, 128), (3, 128), (31, 32), (4, 128), (16, 128), (24, 128), (25, 128)])
@pytest.mark.parametrize("shape", [CacheShape.FLASH, CacheShape.FLASHINFER])
@pytest.mark.parametrize("layers", [1, 40])
def test_expansion_of_any_tile(ops, heads, dim, shape, layers):
    blocks = 12
    src_l = AttnLayout(CacheShape.FLASHINFER, blocks, 16, heads, dim, 1, mx_scaled=True)
    dst_l = AttnLayout(shape, blocks, 16, heads, dim, 2)
    gen = torch.Generator(device=DEV).manual_seed(heads * 1000 + dim)
    src = []
    for _ in range(layers):
        t = src_l.alloc(DEV)
        t.copy_(torch.randint(0, 0x7F, t.shape, dtype=torch.uint8, device=DEV, generator=gen))       # no NaN codes
        sc = src_l.scale_view(t)
        sc.copy_(torch.randint(100, 140, sc.shape, dtype=torch.uint8, device=DEV, generator=gen))
        src.append(t)
    dst = [dst_l.alloc(DEV) for _ in range(layers)]
    x = AttnTransfer(src_l, dst_l, [t.data_ptr() for t in src], [t.data_ptr() for t in dst], DEV, mode=MODE_MXFP8_TO_BF16)
    chunks = [ReqChunk([3, 1, 7], [8, 0, 2], 5, 38, pad_tail=True), ReqChunk([4], [11], 0, 16), ReqChunk([5], [6], 15, 1)]
    x.launch(x.plan(chunks))
    torch.cuda.synchronize()
    assert x.check_status() == (0, 0)
    for s, d in zip(src[:2] + src[-1:], dst[:2] + dst[-1:]):
        want = torch.zeros_like(d)
        reference_transfer(src_l, dst_l, s, want, chunks, None, MODE_MXFP8_TO_BF16)
        assert torch.equal(d, want)
