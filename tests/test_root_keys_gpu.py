"""Key layout and keys of the first coordinates in one launch, against whole-number arithmetic: every number of
dimensions, rows on and off a 16-byte boundary, and row counts around which the grid changes size."""
import pytest
import torch

from minuet_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("ndim", [1, 2, 3, 4])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,clouds", [(1, 1), (5, 3), (1023, 1), (40_001, 4), (606_207, 1), (606_209, 2), (3_031_043, 1)])
def test_against_whole_numbers(ndim, offset, n, clouds):
    gen = torch.Generator(device=DEV).manual_seed(n + ndim)
    flat = torch.randint(-900, 700, (n * ndim + offset,), generator=gen, device=DEV, dtype=torch.int32)
    coords = flat[offset:].view(n, ndim)
    starts, cloud = None, torch.zeros(n, dtype=torch.int64, device=DEV)
    if clouds > 1:
        cuts = [n * k // clouds for k in range(1, clouds)]
        starts = torch.tensor([0, *cuts, n], device=DEV)
        for at in cuts:
            cloud[at:] += 1
    margin = 17
    layout, keys = _lib.host().root_keys(coords, starts, clouds, margin)
    want, shift = torch.zeros(n, dtype=torch.int64, device=DEV), 0
    for k in reversed(range(ndim)):
        low, high = int(coords[:, k].min()) - margin, int(coords[:, k].max()) + margin
        want += (coords[:, k].long() - low) << shift
        shift += (high - low).bit_length()
    assert layout.margin == margin and torch.equal(keys, want + (cloud << shift))
