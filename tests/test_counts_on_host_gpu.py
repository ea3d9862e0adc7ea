"""The row counts and cloud starts that a strided level and a voxelisation bring back: written to host
memory by the kernel where they fit the buffer (1024 values: 1020 clouds), copied beyond."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("clouds", [1, 2, 1019, 1020, 1021, 1500])
def test_counts_and_cloud_starts(clouds):
    rng = np.random.default_rng(clouds)
    per_cloud = [np.unique(rng.integers(-9, 9, (int(rng.integers(1, 40)), 3)), axis=0) for _ in range(clouds)]
    starts = np.cumsum([0] + [len(c) for c in per_cloud])
    coords = torch.as_tensor(np.concatenate(per_cloud), dtype=torch.int32, device=DEV)
    bounds = torch.as_tensor(starts, device=DEV) if clouds > 1 else None
    want = [np.unique(c // 2 * 2, axis=0) for c in per_cloud]
    want_starts = np.cumsum([0] + [len(c) for c in want])
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    out, stride, out_bounds = cache.get_target_coordinates(coords, bounds, 1, 2)
    assert stride == (2, 2, 2) and np.array_equal(out.cpu().numpy(), np.concatenate(want))
    if clouds > 1:
        assert np.array_equal(out_bounds.cpu().numpy(), want_starts)
    sizes = cache.get_kernel_map(coords, 1, bounds, out, stride, out_bounds, 2, 1)[3]
    assert int(sizes.sum()) == len(coords)                    # every voxel has one parent
    # the same counts from points, the means on the way when the host goes on
    points = coords.float() + 0.5
    features = torch.rand(len(coords), 5, device=DEV)
    result = F.voxelize(points, 2.0, batch_dims=bounds, features=features, return_inverse=True)
    voxels, inverse, means = result[0], result[-2], result[-1]
    assert np.array_equal(voxels.cpu().numpy() * 2, np.concatenate(want))
    ref = torch.zeros(len(voxels), 5, device=DEV, dtype=torch.float64).index_add_(0, inverse, features.double())
    ref /= torch.bincount(inverse, minlength=len(voxels))[:, None]
    assert float((means - ref).abs().max()) < 8 * 2.0 ** -23   # at most eight values below one
