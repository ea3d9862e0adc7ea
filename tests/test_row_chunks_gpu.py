"""Row order of large neighbour tables: by hit word inside chunks of rows, at both ends of the rule
that makes the chunks; the order is checked against a stable sort, the layer bit for bit against
the table in the rows' own order."""
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import engine
from minuet_b200.nn.functional import convolution as conv_mod

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,spacing,shift", [
    ((1 << 19) - 1, 1, 31), (1 << 19, 1, 17), ((1 << 19) + 1, 1, 17), ((1 << 22) + 1, 1, 18),
    (1 << 19, 2, 31)])                        # spacing 2: one pair a row
def test_rows_are_sorted_inside_chunks(n, spacing, shift):
    gen = torch.Generator(device=DEV).manual_seed(n)
    i = torch.arange(n + n // 4 + 4096, device=DEV)           # a block with holes
    i = i[torch.randperm(len(i), generator=gen, device=DEV)[:n]].sort().values
    coords = (torch.stack([i >> 14, (i >> 7) & 127, i & 127], 1) * spacing).int()
    bounds = torch.tensor([0, n], device=DEV)
    conv = minuet.nn.SparseConv3d(8, 16, 3, dtype=torch.float16, device=DEV).eval()
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm="implicit")
    sm, tm, _, sizes = cache.get_kernel_map(coords, 1, bounds, coords, 1, bounds, 3, 1)
    _, tile_bits, perm = engine.neighbor_table(sm, tm, engine.host_copy(sizes))

    words = engine.hit_bits(tm).long()
    key = sum(((words >> b) & 1) << (26 - b) for b in range(27))     # rare offsets on top
    for s in (1, 2, 4, 8, 16):                                       # rank in Gray order
        key ^= key >> s
    key |= (torch.arange(n, device=DEV) >> shift) << 27
    assert torch.equal(perm.long(), torch.sort(key, stable=True).indices)
    rows = torch.cat([words[perm.long()], words.new_zeros(-n % 128)]).view(-1, 128)
    for b in range(27):
        assert torch.equal((tile_bits >> b) & 1, ((rows >> b) & 1).amax(1).int())

    x = minuet.SparseTensor(torch.randn(n, 8, generator=gen, device=DEV).half(), coords, batch_dims=bounds)
    with torch.no_grad():
        got = conv(x).F
        conv_mod.REORDER_ROWS = False
        try:
            want = conv(x).F
        finally:
            conv_mod.REORDER_ROWS = True
    assert torch.equal(got, want)      # the same sums in the same order, other rows per tile


@pytest.mark.parametrize("c_in,c_out", [(32, 16), (128, 256)])
def test_first_pass_on_a_fresh_table(c_in, c_out):
    """The first launch after a table was built finds it, and the features, in no cache."""
    gen = torch.Generator(device=DEV).manual_seed(c_in)
    c = torch.unique(torch.randint(0, 72, (60_000, 3), generator=gen, device=DEV, dtype=torch.int32), dim=0)
    bounds = torch.tensor([0, len(c)], device=DEV)
    conv = minuet.nn.SparseConv3d(c_in, c_out, 3, dtype=torch.float16, device=DEV).eval()
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm="implicit")
    feats = torch.randn(len(c), c_in, generator=gen, device=DEV).half()
    want = None
    with torch.no_grad():
        for _ in range(60):
            cache.reset()
            got = conv(minuet.SparseTensor(feats.clone(), c, batch_dims=bounds)).F
            want = got if want is None else want
            assert torch.equal(got, want)
