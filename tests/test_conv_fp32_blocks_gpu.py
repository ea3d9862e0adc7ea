"""Every block shape of the fused fp32 forward, at ragged row counts, with more offsets in a tile than a
block looks at at a time and with tiles of one offset: the bits of gather - FFMA GEMM - scatter."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import engine, synth
from test_conv_fp32_gpu import explicit

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,c_in,c_out,fill", [
    (151_700, 4, 8, 0.3),       # 128 x 32 sums a block
    (152_001, 16, 32, 0.002),   # the same, tiles of one offset
    (80_003, 20, 36, 0.3),      # 64 x 64
    (80_003, 17, 40, 0.002),    # the same, channels that are no multiple of 4
    (40_001, 8, 24, 0.3),       # 64 x 32
    (40_001, 7, 30, 0.01),
    (12_345, 33, 31, 0.3),      # 32 x 32
    (95, 64, 33, 0.5)])         # 32 x 32, eight warps
def test_block_shapes(n, c_in, c_out, fill):
    rng = np.random.default_rng(n)
    src, _ = synth.random_small_batch(rng, 1, n, max(3, round((n / fill) ** (1 / 3))))
    x = torch.as_tensor(rng.standard_normal((len(src), c_in)).astype(np.float32), device=DEV)
    conv = minuet.nn.SparseConv3d(c_in, c_out, 3, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    c = torch.as_tensor(src, device=DEV)
    out = conv(minuet.SparseTensor(x, c)).F
    sm, tm, order, sizes = cache.get_kernel_map(c, 1, None, c, 1, None, 3, 1)
    assert torch.equal(out, explicit(x, conv.kernel.detach(), sm, tm, order, engine.host_copy(sizes), True))
