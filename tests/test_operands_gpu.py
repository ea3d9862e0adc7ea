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
