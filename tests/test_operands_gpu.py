"""Operands that a kernel would follow to memory it cannot reach are refused on the host: nothing is
launched, and the next call works."""
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _points(n=500):
    return torch.rand(n, 3, generator=torch.Generator(device=DEV).manual_seed(n), device=DEV) * 20


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
def test_cloud_starts_on_the_host_are_refused(dtype):
    points, starts = _points().to(dtype), torch.tensor([0, 200, 500])
    with pytest.raises(NotImplementedError):
        F.voxelize(points, 0.5, batch_dims=starts)
    with pytest.raises(NotImplementedError):
        F.voxelize(points, 0.5, batch_dims=starts, features=_points())
    with pytest.raises(NotImplementedError):
        F.voxelize(points, 0.5, features=_points().cpu())
    F.voxelize(points, 0.5, batch_dims=starts.to(DEV))
    torch.cuda.synchronize()


def test_cloud_starts_of_maps_on_the_host_are_refused():
    coords, starts = torch.unique(_points().int(), dim=0), torch.tensor([0, 10, 20])
    cache = lambda: minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    with pytest.raises(NotImplementedError):
        cache().get_target_coordinates(coords, starts, 1, 2)
    with pytest.raises(NotImplementedError):
        cache().get_kernel_map(coords, 1, starts, coords, 1, starts, 3, 1)
    cache().get_kernel_map(coords, 1, None, coords, 1, None, 3, 1)
    torch.cuda.synchronize()


@pytest.mark.needs_grad
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_layer_operands_on_the_host_are_refused(dtype):
    coords = torch.unique(_points().int(), dim=0)
    n = len(coords)
    conv = minuet.nn.SparseConv3d(16, 16, 3, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    x = minuet.SparseTensor(torch.randn(n, 16, device=DEV).to(dtype), coords)
    w, w_t = conv.kernel.detach(), F.transpose_weights(conv.kernel.detach())
    maps = cache.get_kernel_map(coords, 1, None, coords, 1, None, 3, 1)
    sm, tm, order, sizes = maps
    ones = torch.ones(16)
    good = dict(sources=x.F, weights=w, source_masks=sm, target_masks=tm, kernel_map_order=order,
                kernel_map_sizes=sizes, gather_tile_size=1, scatter_tile_size=1)
    for name in ("weights", "source_masks", "target_masks", "kernel_map_order"):
        with pytest.raises(NotImplementedError):
            F.sparse_convolution_forward(**{**good, name: good[name].cpu()})
    with pytest.raises(NotImplementedError):      # the differentiable call
        F.sparse_convolution_forward(**{**good, "sources": x.F.clone().requires_grad_(), "weights": w.cpu()})
    with torch.no_grad():
        for extra in (dict(scale=ones), dict(shift=ones), dict(residual=torch.zeros(n, 16, dtype=dtype))):
            with pytest.raises(NotImplementedError):
                conv.forward_fused(x, **extra)
            with pytest.raises(NotImplementedError):
                F.dense_forward(x.F, w[0], **extra)
        with pytest.raises(NotImplementedError):
            F.dense_forward(x.F, w[0].cpu())
        with pytest.raises(RuntimeError):         # shorter than the row: read past its end
            conv.forward_fused(x, scale=ones[:8].to(DEV))
        with pytest.raises(RuntimeError):
            F.dense_forward(x.F, w[0], residual=torch.zeros(n - 1, 16, dtype=dtype, device=DEV))
        with pytest.raises(RuntimeError):
            F.dense_forward(x.F, w[0, :8])
        if w_t is not None:
            with pytest.raises(NotImplementedError):
                F.sparse_convolution_forward(**good, weights_t=w_t.cpu())
            with pytest.raises(RuntimeError):
                F.sparse_convolution_forward(**good, weights_t=w_t[:5])
        assert torch.equal(F.sparse_convolution_forward(**good, weights_t=w_t), conv(x).F)
    torch.cuda.synchronize()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kernel,stride", [(3, 1), (2, 2)])
def test_a_residual_off_a_16_byte_boundary_on_pair_lists(dtype, kernel, stride):
    gen = torch.Generator(device=DEV).manual_seed(4)
    coords = torch.unique(_points(3000).int(), dim=0)
    conv = minuet.nn.SparseConv3d(16, 24, kernel, stride=stride, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm="explicit")
    x = minuet.SparseTensor(torch.randn(len(coords), 16, generator=gen, device=DEV).to(dtype), coords)
    residual = torch.randn(len(conv(x).F), 24, generator=gen, device=DEV).to(dtype)
    want = conv.forward_fused(x, residual=residual, relu=True).F
    for shift in (1, 2, 4):
        off = torch.empty(residual.numel() + shift, dtype=dtype, device=DEV)[shift:].view_as(residual).copy_(residual)
        assert torch.equal(conv.forward_fused(x, residual=off, relu=True).F, want)
