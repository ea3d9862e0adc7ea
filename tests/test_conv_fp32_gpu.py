"""The fused fp32 forward against gather - FFMA GEMM - scatter of the same library, which sums in
the same order: the same bits, at remainders of the row, channel and offset blocks, with the
offsets of a tile in one block and spread over the blocks of a cluster."""
import ctypes

import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def explicit(x, w, sm, tm, order, sizes, shortcut):
    lib = _lib.load()
    (O, S), T = sm.shape, tm.shape[1]
    out = torch.empty((T, w.shape[2]), device=DEV)
    nbytes = lib.mn_conv_workspace_bytes(engine.np_ptr(sizes), O, S, T, w.shape[1], w.shape[2], _lib.MN_F32,
                                         int(shortcut), 1, -1.0)
    ws = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=DEV)
    _lib.check(lib.mn_sparse_convolution_forward(
        S, T, O, w.shape[1], w.shape[2], _lib.MN_F32, engine.ptr(x), engine.ptr(w), engine.ptr(sm),
        engine.ptr(tm), engine.ptr(order), engine.np_ptr(sizes), 1, 1, int(shortcut), 1, -1.0,
        engine.ptr(out), engine.ptr(engine.status_word(DEV)), engine.ptr(ws), ctypes.c_size_t(ws.numel()),
        engine.stream_ptr(torch.device(DEV))))
    return out


@pytest.mark.parametrize("n,c_in,c_out,kernel,stride", [
    (1, 1, 1, 3, 1), (33, 3, 5, 3, 1), (129, 32, 32, 3, 1), (3000, 33, 33, 3, 1), (20_000, 32, 20, 3, 1),
    (30_000, 64, 64, 3, 1), (2500, 100, 130, 3, 2), (5000, 16, 96, 2, 2), (800, 256, 256, 3, 1)])
def test_same_bits_as_gather_gemm_scatter(n, c_in, c_out, kernel, stride):
    rng = np.random.default_rng(n)
    src, _ = synth.random_small_batch(rng, 1, n, max(2, round((n / 0.25) ** (1 / 3))))
    x = torch.as_tensor(rng.standard_normal((len(src), c_in)).astype(np.float32), device=DEV)
    conv = minuet.nn.SparseConv3d(c_in, c_out, kernel, stride=stride, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    c = torch.as_tensor(src, device=DEV)
    out = conv(minuet.SparseTensor(x, c)).F
    tc, ts, tb = cache.get_target_coordinates(c, None, 1, stride)
    sm, tm, order, sizes = cache.get_kernel_map(c, 1, None, tc, ts, tb, kernel, 1)
    want = explicit(x, conv.kernel.detach(), sm, tm, order, engine.host_copy(sizes), stride == 1)
    assert torch.equal(out, want)
    scale, shift = torch.rand(c_out, device=DEV) + 0.5, torch.rand(c_out, device=DEV)
    res = torch.randn(len(tc), c_out, device=DEV)
    fused = conv.forward_fused(minuet.SparseTensor(x, c), scale=scale, shift=shift, residual=res, relu=True).F
    # product, scale, shift, residual: one rounding each, or fused multiply-adds
    ref = torch.relu(want.double() * scale + shift + res)
    bound = 2.0 ** -22 * ((want * scale).abs() + shift.abs() + res.abs()) + 1e-30
    assert bool(((fused.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("n,c_in,c_out", [(900, 16, 24), (60_000, 16, 24), (20_000, 8, 70)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_weights_that_are_not_finite_reach_their_pairs_only(n, c_in, c_out, value):
    rng = np.random.default_rng(n)
    src, _ = synth.random_small_batch(rng, 1, n, max(2, round((n / 0.25) ** (1 / 3))))
    c = torch.as_tensor(src, device=DEV)
    x = torch.as_tensor(rng.standard_normal((len(src), c_in)).astype(np.float32), device=DEV)
    conv = minuet.nn.SparseConv3d(c_in, c_out, 3, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    sm, tm, order, sizes = cache.get_kernel_map(c, 1, None, c, 1, None, 3, 1)
    clean = conv(minuet.SparseTensor(x, c)).F
    conv.kernel[5, 3, 4] = value
    out = conv(minuet.SparseTensor(x, c)).F
    row = int((order == 5).nonzero())                   # mask row of offset 5
    hit = tm[row] >= 0
    assert bool(hit.any()) and not bool(hit.all())
    bad = torch.zeros_like(out, dtype=torch.bool)
    bad[hit, 4] = True                                  # no feature is zero: inf or NaN in every one
    assert torch.equal(~torch.isfinite(out), bad)
    assert torch.equal(out[~bad], clean[~bad])
    assert torch.equal(torch.nan_to_num(out), torch.nan_to_num(
        explicit(x, conv.kernel.detach(), sm, tm, order, engine.host_copy(sizes), True)))
