"""The radix sort at the row counts where its tiles change shape, and one row to either side of a tile."""
import pytest
import torch

from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [151_551, 151_552, 151_553, 155_648, 155_649, 1_212_415, 1_212_416, 1_212_417])
@pytest.mark.parametrize("extent", [2, 700])
def test_permutation_is_stable(n, extent):
    gen = torch.Generator(device=DEV).manual_seed(n + extent)
    c = torch.randint(-extent, extent, (n, 3), generator=gen, device=DEV, dtype=torch.int32)
    key = ((c[:, 0].long() + extent) * 2 * extent + c[:, 1] + extent) * 2 * extent + c[:, 2] + extent
    got = F.arg_sort_coordinates(c, dtype=torch.int64)
    assert torch.equal(got, torch.sort(key, stable=True).indices)
