"""Weights read as they are (N-major tiles), transposed by the call (off a 16-byte boundary) and
transposed once give the same bits: the same products in the same order."""
import pytest
import torch

import minuet_b200 as minuet

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("c_in,c_out", [(8, 8), (32, 24), (72, 64), (64, 72), (128, 136), (40, 256)])
@pytest.mark.parametrize("rows", [100, 80_001])         # with 80 001 rows: above two tiles per CTA
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_weight_layouts_give_the_same_bits(c_in, c_out, rows, dtype):
    gen = torch.Generator(device=DEV).manual_seed(c_in + c_out + rows)
    side = int((rows * 6) ** (1 / 3)) + 2
    i = torch.randperm(side ** 3, generator=gen, device=DEV)[:rows].sort().values
    coords = torch.stack([i // (side * side), i // side % side, i % side], 1).int()
    for kernel, stride in ((3, 1), (2, 2)):
        conv = minuet.nn.SparseConv3d(c_in, c_out, kernel, stride=stride, dtype=dtype, device=DEV).eval()
        cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
        minuet.set_kernel_map_cache(conv, cache)
        conv.tunable_config.update(algorithm="implicit")
        x = minuet.SparseTensor(torch.randn(rows, c_in, generator=gen, device=DEV).to(dtype), coords)
        with torch.no_grad():
            as_is = conv(x).F
            aligned = conv.kernel.data
            shifted = torch.empty(aligned.numel() + 4, dtype=dtype, device=DEV)[4:].view_as(aligned)
            conv.kernel.data = shifted.copy_(aligned)           # 8 bytes off
            off = conv(x).F
            conv.kernel.data = aligned
            conv.freeze_weights()
            frozen = conv(x).F
        assert torch.equal(as_is, frozen) and torch.equal(off, frozen)
