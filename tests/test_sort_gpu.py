"""The radix sort and what is built on it, at the sizes where it can go wrong: one key, tile
remainders, the switch between tile sizes, keys that share every digit, indices that no longer fit
below the key; voxelisation against numpy."""
import numpy as np
import pytest
import torch

from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,extent,clouds", [
    (1, 1, 1), (33, 4, 1), (1023, 50, 1), (1025, 1, 1), (4097, 7, 3), (606_207, 300, 1), (606_208, 5, 2),
    (1_000_003, 2000, 5), (70_000, 2 ** 20, 1)])
def test_arg_sort_is_the_stable_permutation(n, extent, clouds):
    gen = torch.Generator(device=DEV).manual_seed(n)
    c = torch.randint(-extent, extent + 1, (n, 3), generator=gen, device=DEV, dtype=torch.int32)
    bounds = None
    cloud = torch.zeros(n, dtype=torch.int64, device=DEV)
    if clouds > 1:
        cuts = sorted(int(n * f) for f in np.random.default_rng(n).random(clouds - 1))
        bounds = torch.tensor([0, *cuts, n], device=DEV)
        for b in cuts:
            cloud[b:] += 1
    got = F.arg_sort_coordinates(c, batch_dims=bounds, dtype=torch.int64)
    want = torch.arange(n, device=DEV)
    for key in (c[:, 2], c[:, 1], c[:, 0], cloud):          # least significant first, each stable
        want = want[torch.sort(key[want], stable=True).indices]
    assert torch.equal(got, want)
    assert torch.equal(F.arg_sort_coordinates(c, batch_dims=bounds, dtype=torch.int64,
                                              enable_flattening=False), want)


@pytest.mark.parametrize("n,ndim,dtype,channels,fdtype", [
    (1, 3, torch.float32, 1, torch.float32), (1000, 2, torch.float64, 9, torch.float32),
    (4097, 3, torch.float32, 4, torch.float16), (200_001, 3, torch.float32, 6, torch.float32),
    (5000, 3, torch.float64, 130, torch.bfloat16)])
def test_voxelize_against_numpy(n, ndim, dtype, channels, fdtype):
    rng = np.random.default_rng(n)
    points = torch.as_tensor(rng.uniform(-7, 9, (n, ndim)), device=DEV).to(dtype)
    feats = torch.as_tensor(rng.standard_normal((n, channels)), device=DEV).to(fdtype)
    size = 0.3 if ndim == 3 else [0.3, 0.02]
    half = n // 3
    bounds = torch.tensor([0, half, n], device=DEV)
    voxels, starts, inverse, means = F.voxelize(points, size, batch_dims=bounds, return_inverse=True,
                                                features=feats)
    p = points.cpu().numpy()
    cells = np.floor(p / np.asarray(size, dtype=p.dtype)).astype(np.int64)
    rows = np.concatenate([(np.arange(n) >= half).astype(np.int64)[:, None], cells], axis=1)
    want, inv = np.unique(rows, axis=0, return_inverse=True)
    inv = inv.reshape(-1)
    assert voxels.dtype == torch.int32 and np.array_equal(voxels.cpu().numpy(), want[:, 1:])
    assert np.array_equal(inverse.cpu().numpy(), inv)
    assert starts.tolist() == [0, int((want[:, 0] == 0).sum()), len(want)]
    f = feats.double().cpu().numpy()
    count = np.bincount(inv, minlength=len(want))
    total, size_ = np.zeros((len(want), channels)), np.zeros((len(want), channels))
    np.add.at(total, inv, f)
    np.add.at(size_, inv, np.abs(f))
    ulp = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[fdtype]
    mean = total / count[:, None]
    # count additions and a product by 1 / count in fp32, one rounding to the feature type
    bound = (count[:, None] + 2) * 2.0 ** -23 * size_ / count[:, None] + ulp * np.abs(mean) + 1e-7
    assert (np.abs(means.double().cpu().numpy() - mean) <= bound).all()
    wide = torch.cat([points, points + 3e8]) if dtype == torch.float64 else None
    if wide is not None and ndim == 3:      # a box whose keys leave no room for the index
        v, inv2 = F.voxelize(wide, size, return_inverse=True)[::2]
        assert len(v) > len(want) and int(inv2.max()) == len(v) - 1
