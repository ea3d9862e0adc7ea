"""The fused forward kernel on freshly built tables, many times over: the ring of index blocks that its
producers read (slots handed back and refilled, sub-tiles that lack an offset) against plain torch sums.
Features and weights are small whole numbers, so that every order of the sums gives the same bits."""
import pytest
import torch

import minuet_b200 as minuet

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cloud(gen):
    """A block with most neighbours present, then voxels without any: tiles with all offsets and tiles
    with the centre only, an odd number of them."""
    block = torch.stack(torch.meshgrid(*3 * [torch.arange(18, device=DEV)], indexing="ij"), -1).view(-1, 3)
    block = block[torch.rand(len(block), generator=gen, device=DEV) < 0.8]
    lone = torch.stack(torch.meshgrid(*3 * [torch.arange(14, device=DEV)], indexing="ij"), -1).view(-1, 3) * 3 + 40
    n = (len(block) + len(lone)) // 256 * 256 + 100          # the last pair of tiles is half empty
    c = torch.cat([block, lone])[:n]
    assert (-(-len(c) // 128)) % 2 == 1
    return c.int()


@pytest.mark.parametrize("sub_tiles,c_in,c_out", [(1, 32, 16), (1, 128, 64), (2, 32, 96), (2, 64, 128), (2, 128, 256)])
def test_fresh_tables_give_exact_sums(sub_tiles, c_in, c_out):
    gen = torch.Generator(device=DEV).manual_seed(c_in + c_out)
    coords = _cloud(gen)
    n = len(coords)
    conv = minuet.nn.SparseConv3d(c_in, c_out, 3, dtype=torch.float16, device=DEV).eval()
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm="implicit", sub_tiles=sub_tiles)
    conv.kernel.copy_(torch.randint(-1, 2, conv.kernel.shape, generator=gen, device=DEV))
    x = torch.randint(-1, 2, (n, c_in), generator=gen, device=DEV).half()
    sm, tm, order, _ = cache.get_kernel_map(coords, 1, None, coords, 1, None, 3, 1)
    want = torch.zeros(n, c_out, device=DEV)
    for p in range(27):
        s, t = (torch.nonzero(m[p] >= 0)[:, 0] for m in (sm, tm))
        s, t = s[sm[p, s].argsort()], t[tm[p, t].argsort()]
        want[t] += x[s].float() @ conv.kernel[order[p].long()].float()     # rows of a mask row are distinct
    assert float(want.abs().max()) < 2048                        # exact in 16 bits
    for _ in range(400):
        cache.reset()
        got = conv(minuet.SparseTensor(x.clone(), coords)).F
        assert torch.equal(got.float(), want)
