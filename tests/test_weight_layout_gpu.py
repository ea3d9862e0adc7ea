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


@pytest.mark.needs_grad
@pytest.mark.parametrize("kernel,stride", [(3, 1), (2, 2)])
@pytest.mark.parametrize("algorithm", ["implicit", "explicit"])
def test_gradients_of_a_weight_off_a_16_byte_boundary(kernel, stride, algorithm):
    """A weight that is a view into a flat parameter buffer trains like any other."""
    gen = torch.Generator(device=DEV).manual_seed(1)
    i = torch.randperm(20 ** 3, generator=gen, device=DEV)[:3000].sort().values
    coords = torch.stack([i // 400, i // 20 % 20, i % 20], 1).int()
    conv = minuet.nn.SparseConv3d(32, 48, kernel, stride=stride, dtype=torch.float16, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm=algorithm)
    x = torch.randn(3000, 32, generator=gen, device=DEV).half().requires_grad_()
    aligned = conv.kernel.data
    results = []
    for shift in (0, 1, 4):
        flat = torch.empty(aligned.numel() + shift, dtype=torch.float16, device=DEV)
        conv.kernel.data = flat[shift:].view_as(aligned).copy_(aligned)
        out = conv(minuet.SparseTensor(x, coords)).F
        results.append((out, *torch.autograd.grad(out, (x, conv.kernel), torch.ones_like(out))))
    for off in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], off))
    w_t = minuet.nn.functional.transpose_weights(aligned)
    off = torch.empty(w_t.numel() + 1, dtype=torch.float16, device=DEV)[1:].view_as(w_t).copy_(w_t)
    maps = conv._lookup(minuet.SparseTensor(x, coords))[3:7]
    with torch.no_grad():
        got = minuet.nn.functional.sparse_convolution_forward(
            x, aligned, *maps, 1, 1, allow_shortcut_matmul=conv._allow_shortcut_matmul, algorithm=algorithm,
            weights_t=off)
    assert torch.equal(got, results[0][0])
