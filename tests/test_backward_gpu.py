"""Weight gradients against float64 sums over the oracle's pairs, at the sizes where the kernels
can go wrong: one pair and none per offset, remainders of the 64-pair and 64-channel blocks, more
channels than one block holds, channel counts the tensor cores do not take."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import synth
from minuet_b200.utils.helpers import generate_kernel_offsets

pytestmark = [pytest.mark.gpu, pytest.mark.needs_grad]
DEV = "cuda:0"
ROUND = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("n,c_in,c_out,dtype,kernel", [
    (1, 8, 8, torch.float16, 3), (65, 64, 64, torch.float16, 3), (1500, 72, 136, torch.float16, 3),
    (3000, 256, 256, torch.bfloat16, 2), (700, 320, 16, torch.float16, 3), (900, 12, 20, torch.float16, 3),
    (1, 3, 5, torch.float32, 3), (2000, 33, 65, torch.float32, 3), (4000, 32, 64, torch.float32, 3),
    (800, 128, 32, torch.float32, 5)])
def test_weight_gradient(oracle_lib, n, c_in, c_out, dtype, kernel):
    rng = np.random.default_rng(n + c_in)
    src, _ = synth.random_small_batch(rng, 1, n, max(2, round((n / 0.3) ** (1 / 3))))
    off = generate_kernel_offsets(3, kernel, 1, 1).astype(np.int32)
    km = oracle_lib.build_kernel_map(src, src, off)["kernel_map"]
    x = torch.as_tensor(rng.standard_normal((len(src), c_in)), device=DEV).to(dtype)
    g = torch.as_tensor(rng.standard_normal((len(src), c_out)), device=DEV).to(dtype)
    conv = minuet.nn.SparseConv3d(c_in, c_out, kernel, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    out = conv(minuet.SparseTensor(x, torch.as_tensor(src, device=DEV))).F
    (dw,) = torch.autograd.grad(out, (conv.kernel,), g)
    for o in range(len(off)):
        t = torch.as_tensor(np.nonzero(km[o] >= 0)[0], device=DEV)
        s = torch.as_tensor(km[o][km[o] >= 0].astype(np.int64), device=DEV)
        a, b = x[s].double(), g[t].double()
        want = a.t() @ b
        # m additions in fp32 (the tensor cores may truncate: 2^-23 each), one rounding at the end
        bound = (len(t) + 2) * 2.0 ** -23 * (a.abs().t() @ b.abs()) + ROUND[dtype] * want.abs() + 1e-7
        assert bool(((dw[o].double() - want).abs() <= bound).all()), (o, len(t))
    (again,) = torch.autograd.grad(conv(minuet.SparseTensor(x, torch.as_tensor(src, device=DEV))).F,
                                   (conv.kernel,), g)
    assert torch.equal(dw, again)


@pytest.mark.parametrize("kernel", [1, 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("create_graph", [False, True])
def test_a_gradient_that_torch_keeps_without_memory(kernel, dtype, create_graph):
    """The gradient of sgn is zero, and a tensor that has no memory."""
    rng = np.random.default_rng(3)
    src, _ = synth.random_small_batch(rng, 1, 3000, 24)
    assert len(src) >= 1024
    conv = minuet.nn.SparseConv3d(16, 24, kernel, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    x = torch.ones(len(src), 16, device=DEV, dtype=dtype, requires_grad=True)
    seen = []
    out = conv(minuet.SparseTensor(x, torch.as_tensor(src, device=DEV))).F
    out.register_hook(lambda g: seen.append(g._is_zerotensor()))
    grads = torch.autograd.grad(torch.sgn(out).sum(), (x, conv.kernel), create_graph=create_graph)
    assert seen == [True]
    for grad, of in zip(grads, (x, conv.kernel)):
        assert grad.shape == of.shape and grad.dtype == dtype and bool((grad == 0).all())
