"""torch.jit.trace sees nothing of the native calls: it is refused instead of recording their results as
constants."""
import warnings

import pytest
import torch

import minuet_b200 as minuet

pytestmark = [pytest.mark.gpu, pytest.mark.needs_grad]
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("kernel,grad", [(3, True), (3, False), (1, False)])
def test_tracing_is_refused(dtype, kernel, grad):
    coords = torch.stack(torch.meshgrid(*3 * [torch.arange(4, device=DEV)], indexing="ij"), -1).view(-1, 3).int()
    conv = minuet.nn.SparseConv3d(8, 8, kernel, dtype=dtype, device=DEV).requires_grad_(grad)
    minuet.set_kernel_map_cache(conv, minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV))
    x = torch.randn(64, 8, device=DEV).to(dtype)
    call = lambda features: conv(minuet.SparseTensor(features, coords)).F
    with torch.set_grad_enabled(grad), warnings.catch_warnings():
        warnings.simplefilter("ignore")
        call(x)
        with pytest.raises(RuntimeError, match="trace"):
            torch.jit.trace(call, (x,), check_trace=False)
        call(x)
