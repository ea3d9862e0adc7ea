"""Weight gradients against fp64 sums over the pairs: tiles of 64 and 32 channels, channels that are no
multiple of 4, one pair, ragged pair counts and one offset with many items (several runs in the
reduction), to rounding; and to the bit where features and gradients are small whole numbers, so that a
pair, an item or a run that is lost or taken twice shows."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


CASES = pytest.mark.parametrize("n,c_in,c_out,fill,dtype", [
    (1, 4, 4, 0.5, torch.float32), (129, 64, 64, 0.4, torch.float32), (2000, 36, 100, 0.3, torch.float32),
    (2000, 100, 20, 0.3, torch.float32), (700, 33, 5, 0.4, torch.float32), (60_000, 8, 8, 0.005, torch.float32),
    (60_000, 64, 68, 0.005, torch.float32), (900, 20, 37, 0.3, torch.float16), (60_000, 16, 24, 0.005, torch.bfloat16),
    (60_000, 63, 61, 0.005, torch.float32), (60_000, 61, 35, 0.005, torch.float16)])


def gradient(n, c_in, c_out, fill, dtype, values):
    """Features, output gradients, the weights' gradient per mask row and the pairs of every mask row."""
    rng = np.random.default_rng(n + c_in)
    src, _ = synth.random_small_batch(rng, 1, n, max(2, round((n / fill) ** (1 / 3))))
    c = torch.as_tensor(src, device=DEV)
    conv = minuet.nn.SparseConv3d(c_in, c_out, 3, device=DEV, dtype=dtype)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    x = torch.as_tensor(values(rng, (len(src), c_in)), device=DEV).to(dtype)
    g = torch.as_tensor(values(rng, (len(src), c_out)), device=DEV).to(dtype)
    with torch.enable_grad():
        got, = torch.autograd.grad(conv(minuet.SparseTensor(x, c)).F, (conv.kernel,), g)
    sm, tm, order, _ = cache.get_kernel_map(c, 1, None, c, 1, None, 3, 1)
    pairs = []
    for p in range(len(order)):
        s, t = (sm[p] >= 0).nonzero()[:, 0], (tm[p] >= 0).nonzero()[:, 0]
        pairs.append((s[sm[p][s].argsort()], t[tm[p][t].argsort()]))
    return x.double(), g.double(), got[order.long()], pairs


@CASES
def test_against_fp64(n, c_in, c_out, fill, dtype):
    x, g, got, pairs = gradient(n, c_in, c_out, fill, dtype, lambda rng, shape: rng.standard_normal(shape))
    # sums of `pairs` exact or once rounded products in fp32, in any order, then one rounding
    half_ulp = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    for p, (s, t) in enumerate(pairs):
        a, b = x[s], g[t]
        ref, size = a.t() @ b, a.abs().t() @ b.abs()
        bound = (len(s) + 1) * 2.0 ** -24 * size + half_ulp * ref.abs() + 1e-7
        assert bool(((got[p].double() - ref).abs() <= bound).all())


@CASES
def test_whole_numbers_exactly(n, c_in, c_out, fill, dtype):
    x, g, got, pairs = gradient(n, c_in, c_out, fill, dtype, lambda rng, shape: rng.integers(-3, 4, shape))
    # every partial sum is a whole number below 9 * 60 000 < 2^24: exact in fp32, in any order; then one rounding
    for p, (s, t) in enumerate(pairs):
        assert torch.equal(got[p], (x[s].t() @ g[t]).to(dtype)), p
