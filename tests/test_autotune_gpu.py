"""The autotuner times what a layer runs."""
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,channels,kernel,stages,sub_tiles", [
    (torch.float32, 8, 3, False, set()),           # one kernel
    (torch.float32, 4, 5, True, set()),            # 125 offsets: gather, GEMM, scatter
    (torch.float16, 3, 3, True, set()),            # channels that the tensor-core paths do not take
    (torch.float16, 16, 3, False, {0, 1, 2})])     # pair lists and the fused kernel
def test_what_is_timed(monkeypatch, dtype, channels, kernel, stages, sub_tiles):
    timed, subs = set(), set()
    for name in ("cuda_time_gather", "cuda_time_gemm", "cuda_time_scatter"):
        monkeypatch.setattr(F, name, lambda *a, _n=name, **k: timed.add(_n) or 1.0)
    whole = F.time_forward
    monkeypatch.setattr(F, "time_forward", lambda *a, **k: subs.add(k["sub_tiles"]) or whole(*a, **k))
    monkeypatch.setattr(minuet.nn.SparseConv, "__NUM_TUNING_ROUNDS__", 1)
    coords = torch.stack(torch.meshgrid(*3 * [torch.arange(8, device=DEV)], indexing="ij"), -1).view(-1, 3).int()
    conv = minuet.nn.SparseConv3d(channels, channels, kernel, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    with conv.autotune():
        conv(minuet.SparseTensor(torch.randn(len(coords), channels, device=DEV).to(dtype), coords))
    assert timed == ({"cuda_time_gather", "cuda_time_gemm", "cuda_time_scatter"} if stages else set())
    assert subs == sub_tiles
