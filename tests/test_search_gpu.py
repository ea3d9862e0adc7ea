"""Kernel-map search at the edges of its cells and of its 32-bit keys: groups of offsets that span up to a
whole cell and more, offsets that are not next to one another, boxes whose keys need 64 bits, rows that are
the table and rows that are not, offsets all on one side."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F
from minuet_b200.utils.helpers import generate_kernel_offsets

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cloud(rng, box, n):
    """Clusters (neighbours in every direction) at places all over the box, its corners among them."""
    at = [rng.integers(0, b - 12, size=n // 40) for b in box]
    c = np.stack(at, 1).repeat(40, 0) + rng.integers(0, [min(b, s) for b, s in zip(box, (3, 4, 12))], size=(n // 40 * 40, 3))
    return np.unique(np.concatenate([c, [[0, 0, 0], [b - 1 for b in box]]]), axis=0).astype(np.int32)


@pytest.mark.parametrize("box", [(40, 40, 70), (30, 5000, 3000), (30, 1 << 15, 1 << 15), (1 << 17, 1 << 17, 1 << 17)])
@pytest.mark.parametrize("kernel,dilation", [(3, 1), (2, 1), (3, 2), ((1, 1, 15), 1), ((1, 1, 16), 1), ((1, 2, 16), 1),
                                             ((1, 1, 31), 1), ((1, 1, 5), 7), ((3, 3, 1), 1)])
def test_maps_over_spans_and_boxes(oracle_lib, box, kernel, dilation):
    rng = np.random.default_rng(sum(box) % 1000 + dilation)
    src = _cloud(rng, box, 4000)
    tgt = oracle_lib.downsample(src, 2, None)[0]
    off = generate_kernel_offsets(3, kernel, 1, dilation).astype(np.int32)
    d_src = torch.as_tensor(src, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    for stride, to in ((1, src), (2, tgt)):
        c, s, b = cache.get_target_coordinates(d_src, None, 1, stride)
        assert np.array_equal(c.cpu().numpy(), to)
        sm, tm, order, sizes = cache.get_kernel_map(d_src, 1, None, c, s, b, kernel, dilation)
        want = oracle_lib.build_kernel_map(src, to, off, None, None)
        for got, key in ((sizes, "sorted_sizes"), (order, "order"), (tm, "target_masks"), (sm, "source_masks")):
            assert np.array_equal(got.cpu().numpy(), want[key]), key


@pytest.mark.parametrize("sign", [1, -1])
def test_offsets_on_one_side_of_the_rows_own_place(oracle_lib, sign):
    rng = np.random.default_rng(3)
    src = _cloud(rng, (40, 40, 70), 6000)
    off = sign * np.array([[1, 0, 0], [0, 1, 2], [2, 2, 2], [0, 0, 5], [0, 0, 19], [0, 0, 4]], np.int32)
    d = torch.as_tensor(src, device=DEV)
    got = F.query_sorted_index_with_offsets(d, d, torch.as_tensor(off, device=DEV))
    assert np.array_equal(got.cpu().numpy(), oracle_lib.query(src, src, off))


@pytest.mark.parametrize("shift", [-1000, 1000])
@pytest.mark.parametrize("n", [1, 700])
def test_windows_without_a_key(oracle_lib, shift, n):
    """Targets that all lie before, or behind, every source: no tile has anything to look through."""
    rng = np.random.default_rng(n)
    src = _cloud(rng, (40, 40, 70), 2000)
    tgt = (src[:n] + np.array([shift, 0, 0])).astype(np.int32)
    off = generate_kernel_offsets(3, 3, 1, 1).astype(np.int32)
    d_src, d_tgt = (torch.as_tensor(c, device=DEV) for c in (src, tgt))
    got = F.query_sorted_index_with_offsets(d_src, d_tgt, torch.as_tensor(off, device=DEV))
    assert (got == -1).all()


@pytest.mark.parametrize("z", [255, 256, 257, 258, 259, 300, 319, 320, 321, 322, 323, 400])
def test_windows_as_wide_as_relative_keys_go(oracle_lib, z):
    """Two voxels whose keys are 2^32 - z apart (nine bits of the last dimension): a window is searched by 32-bit
    relative keys up to 2^32 - 258, and its last voxel is found there as beyond."""
    src = np.array([[0, 0, z], [0, 1 << 23, 0]], np.int32)
    off = generate_kernel_offsets(3, 3, 1, 1).astype(np.int32)
    d = torch.as_tensor(src, device=DEV)
    want = oracle_lib.query(src, src, off)
    assert (want >= 0).sum() == 2
    got = F.query_sorted_index_with_offsets(d, d, torch.as_tensor(off, device=DEV))
    assert np.array_equal(got.cpu().numpy(), want)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    sm, tm, _, sizes = cache.get_kernel_map(d, 1, None, d, 1, None, 3, 1)
    assert sizes.cpu().tolist() == [0] * 26 + [2] and sm[26].cpu().tolist() == tm[26].cpu().tolist() == [0, 1]
