"""Every block shape of the fused fp32 forward, alone and in clusters, at the row counts where the dispatch
changes over: with more offsets in a tile than a block looks at at a time, with tiles of one offset, with
channels that can be copied 16 bytes at a time and not.  The bits of gather - FFMA GEMM - scatter,
also with weights that are not finite, and the fused epilogue."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import engine
from test_conv_fp32_gpu import explicit

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 148


def shape_of(rows, c_in, c_out):
    """The dispatch of mn_sparse_convolution_forward_implicit_fp32."""
    columns = -(-c_out // 32)
    tall, mid, low = (-(-rows // r) * columns for r in (128, 64, 32))
    if low <= 48:
        return "cluster of 32 rows"
    if mid <= 55 or (c_in >= 256 and SMS <= 2 * mid and 3 * mid <= 2 * SMS):
        return "cluster of 64 rows"
    if tall >= 8 * SMS:
        return "64 x 64" if columns > 1 else "128 x 32"
    if mid >= 4 * SMS:
        return "64 x 32"
    return "32 x 32" if 2 * low >= 5 * SMS else "eight warps"


DENSE, SPARSE, ONE = 0.9, 0.05, 0.002       # share of the cells that are occupied: 20, 2 and 1 pairs a row


@pytest.mark.parametrize("n,c_in,c_out,fill,shape", [
    (151_425, 4, 8, DENSE, "128 x 32"), (151_500, 7, 30, DENSE, "128 x 32"), (152_001, 16, 32, ONE, "128 x 32"),
    (152_001, 5, 32, ONE, "128 x 32"), (75_649, 20, 36, DENSE, "64 x 64"), (76_003, 17, 40, DENSE, "64 x 64"),
    (80_003, 16, 64, ONE, "64 x 64"), (80_003, 17, 40, ONE, "64 x 64"), (75_648, 4, 33, DENSE, "64 x 32"),
    (37_825, 8, 24, DENSE, "64 x 32"), (40_001, 7, 30, DENSE, "64 x 32"), (40_001, 8, 16, ONE, "64 x 32"),
    (37_824, 8, 24, DENSE, "32 x 32"), (11_809, 33, 31, SPARSE, "32 x 32"), (11_808, 12, 16, DENSE, "eight warps"),
    (5_001, 21, 33, SPARSE, "eight warps"), (3_521, 36, 20, SPARSE, "eight warps"),
    (3_520, 36, 20, DENSE, "cluster of 64 rows"), (1_700, 15, 50, SPARSE, "cluster of 64 rows"),
    (2_400, 256, 64, SPARSE, "cluster of 64 rows"), (49, 8, 1024, DENSE, "cluster of 64 rows"),
    (1_537, 20, 24, SPARSE, "cluster of 64 rows"), (1_536, 20, 24, SPARSE, "cluster of 32 rows"),
    (300, 33, 70, DENSE, "cluster of 32 rows"), (95, 64, 33, SPARSE, "cluster of 32 rows"),
    (33, 256, 128, DENSE, "cluster of 32 rows"), (1, 1, 1, DENSE, "cluster of 32 rows"), (31, 3, 5, ONE, "cluster of 32 rows")])
def test_block_shapes(n, c_in, c_out, fill, shape):
    assert shape_of(n, c_in, c_out) == shape
    rng = np.random.default_rng(n)
    extent = int(np.ceil((n / fill) ** (1 / 3)))
    cells = np.sort(rng.choice(extent ** 3, n, replace=False))
    c = torch.as_tensor(np.stack([cells // extent ** 2, cells // extent % extent, cells % extent], 1).astype(np.int32),
                        device=DEV)
    x = torch.as_tensor(rng.standard_normal((n, c_in)).astype(np.float32), device=DEV)
    conv = minuet.nn.SparseConv3d(c_in, c_out, 3, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    sm, tm, order, sizes = cache.get_kernel_map(c, 1, None, c, 1, None, 3, 1)
    pairs = (tm >= 0).sum(0)
    if fill == DENSE and n > 1000:
        assert int(pairs.max()) > 16              # more offsets than a tall block looks at at a time
    if fill == ONE:
        assert float((pairs == 1).float().mean()) > 0.9
    want = explicit(x, conv.kernel.detach(), sm, tm, order, engine.host_copy(sizes), True)
    assert torch.equal(conv(minuet.SparseTensor(x, c)).F, want)
    scale, shift = torch.rand(c_out, device=DEV) + 0.5, torch.rand(c_out, device=DEV)
    res = torch.randn(n, c_out, device=DEV)
    fused = conv.forward_fused(minuet.SparseTensor(x, c), scale=scale, shift=shift, residual=res, relu=True).F
    # product, scale, shift, residual: one rounding each, or fused multiply-adds
    ref = torch.relu(want.double() * scale + shift + res)
    bound = 2.0 ** -22 * ((want * scale).abs() + shift.abs() + res.abs()) + 1e-30
    assert bool(((fused.double() - ref).abs() <= bound).all())
    # a weight that is not finite reaches the rows that have its offset, and no others
    k = 13 if fill == ONE else 5
    conv.kernel[k, c_in // 2, c_out // 2] = float("inf")
    out = conv(minuet.SparseTensor(x, c)).F
    bad = torch.zeros_like(out, dtype=torch.bool)
    bad[tm[int((order == k).nonzero())] >= 0, c_out // 2] = True       # no feature is zero
    assert torch.equal(~torch.isfinite(out), bad)
    assert torch.equal(out[~bad], want[~bad])
    assert torch.equal(out[bad], explicit(x, conv.kernel.detach(), sm, tm, order, engine.host_copy(sizes), True)[bad])


@pytest.mark.parametrize("n,kernel,stride", [(8, 2, 2), (64, 3, 4), (27, 3, 3), (500, 2, 2)])
def test_many_sources_of_few_targets(n, kernel, stride):
    """Strided layers whose targets have most offsets, on clusters."""
    rng = np.random.default_rng(n)
    extent = int(np.ceil(n ** (1 / 3)))
    cells = np.sort(rng.choice(extent ** 3, n, replace=False))
    c = torch.as_tensor(np.stack([cells // extent ** 2, cells // extent % extent, cells % extent], 1).astype(np.int32),
                        device=DEV)
    x = torch.as_tensor(rng.standard_normal((n, 40)).astype(np.float32), device=DEV)
    conv = minuet.nn.SparseConv3d(40, 72, kernel, stride=stride, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    out = conv(minuet.SparseTensor(x, c)).F
    tc, ts, tb = cache.get_target_coordinates(c, None, 1, stride)
    sm, tm, order, sizes = cache.get_kernel_map(c, 1, None, tc, ts, tb, kernel, 1)
    assert shape_of(len(tc), 40, 72) == "cluster of 32 rows"
    assert torch.equal(out, explicit(x, conv.kernel.detach(), sm, tm, order, engine.host_copy(sizes), False))
