"""Masks of the fused map build against query + sizes + order + masks step by step, around the
128-row units and the ranges of the emission kernel's warps."""
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F
from minuet_b200.utils.helpers import generate_kernel_offsets

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 4097, 300_001, 1_300_000])
@pytest.mark.parametrize("kernel,stride", [(3, 1), (2, 2), (1, 1)])
def test_fused_build_gives_the_stepwise_masks(n, kernel, stride):
    gen = torch.Generator(device=DEV).manual_seed(n)
    side = max(3, int((n * 4) ** (1 / 3)) + 1)
    i = torch.randperm(side ** 3, generator=gen, device=DEV)[:n].sort().values
    coords = torch.stack([i // (side * side), i // side % side, i % side], 1).int()
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    to, to_stride, to_bounds = coords, 1, None
    if stride > 1:
        to, to_stride, to_bounds = cache.get_target_coordinates(coords, None, 1, stride)
    sm, tm, order, sizes = cache.get_kernel_map(coords, 1, None, to, to_stride, to_bounds, kernel, 1)
    offsets = torch.as_tensor(generate_kernel_offsets(3, kernel, 1, 1), dtype=torch.int32, device=DEV)
    m = F.query_sorted_index_with_offsets(coords, to, offsets)
    counts = F.compute_kernel_map_sizes(m)
    want_order = torch.sort(counts, stable=True).indices
    assert torch.equal(order.long(), want_order.long())
    assert torch.equal(sizes.long(), counts[want_order].long())
    want_sm, want_tm = F.compute_kernel_map_masks(len(coords), m[want_order], counts[want_order])
    assert torch.equal(tm, want_tm) and torch.equal(sm, want_sm)
