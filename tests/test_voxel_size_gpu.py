"""Voxel sizes in every form that broadcasts against [N, D] points."""
import numpy as np
import pytest
import torch

from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("size", [
    0.5, [0.5], [0.5, 0.75, 1.25], (0.5, 0.75, 1.25), range(1, 4), np.float64(0.5), np.float32(0.5), np.array(0.5),
    np.array([0.5, 0.75, 1.25]), np.array([[0.5, 0.75, 1.25]]), [[0.5, 0.75, 1.25]], np.full((400, 3), 0.5),
    np.linspace(0.5, 1, 400)[:, None], torch.tensor(0.5), torch.tensor([0.5, 0.75, 1.25]), [torch.tensor(0.5)] * 3],
    ids=lambda s: type(s).__name__ + str(np.shape(s)))
def test_sizes(size):
    gen = torch.Generator(device=DEV).manual_seed(3)
    points = torch.rand(400, 3, generator=gen, device=DEV) * 8
    features = torch.rand(400, 2, generator=gen, device=DEV)
    voxels, _, inverse, means = F.voxelize(points, size, return_inverse=True, features=features)
    cells = torch.floor(points / torch.as_tensor(size, dtype=points.dtype, device=DEV)).int()
    want, run = torch.unique(cells, dim=0, return_inverse=True)
    assert torch.equal(voxels, want) and torch.equal(inverse, run)
    sums = torch.zeros(len(want), 2, dtype=torch.float64, device=DEV).index_add_(0, run, features.double())
    assert torch.allclose(means.double(), sums / torch.bincount(run)[:, None], rtol=1e-5)


@pytest.mark.parametrize("size", ["a", None, [0.5, 0.5], object(), np.zeros((3, 1))])
def test_sizes_that_do_not_broadcast(size):
    with pytest.raises((TypeError, ValueError, RuntimeError)):
        F.voxelize(torch.rand(400, 3, device=DEV), size)
