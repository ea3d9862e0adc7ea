"""The radix sort at the row counts where its tiles change shape, and one row to either side of a tile, with
the index below the key and (63 key bits) in an array of its own."""
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


@pytest.mark.parametrize("n", [151_551, 151_552, 155_649, 1_212_415, 1_212_417])
def test_index_beside_a_full_key(n):
    extent = 2 ** 20
    gen = torch.Generator(device=DEV).manual_seed(n)
    c = torch.randint(-extent, extent, (n, 3), generator=gen, device=DEV, dtype=torch.int32)
    c[n // 2:] = c[:n - n // 2].clone()                    # equal keys far apart
    c[0], c[1] = -extent, extent - 1                       # 21 bits a dimension, whatever was drawn
    got = F.arg_sort_coordinates(c, dtype=torch.int64)
    want = torch.arange(n, device=DEV)
    for d in (2, 1, 0):                                    # least significant first, each stable
        want = want[torch.sort(c[want, d], stable=True).indices]
    assert torch.equal(got, want)


@pytest.mark.parametrize("n", [1_818_623, 1_818_624, 1_818_625, 2_182_348, 2_182_349])
@pytest.mark.parametrize("extent", [2, 700])
def test_permutation_is_stable_where_one_wave_ends(n, extent):
    test_permutation_is_stable(n, extent)


@pytest.mark.parametrize("n", [1_836_810, 1_836_811])
@pytest.mark.parametrize("extent", [2, 700])
def test_permutation_is_stable_a_hundredth_past_one_wave(n, extent):
    test_permutation_is_stable(n, extent)


@pytest.mark.parametrize("n", [1_818_625, 1_836_810, 1_836_811, 2_182_348, 2_182_349, 2_400_000])
def test_index_beside_a_full_key_past_one_wave(n):
    test_index_beside_a_full_key(n)
