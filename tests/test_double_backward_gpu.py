"""Second derivatives of the convolution (gradient penalties, Hessian products) against the same sums of
plain torch in 64 bits."""
import pytest
import torch

import minuet_b200 as minuet

pytestmark = [pytest.mark.gpu, pytest.mark.needs_grad]
DEV = "cuda:0"


def _plain(x, w, sm, tm, order, rows):
    out = x.new_zeros(rows, w.shape[2])
    for p in range(len(sm)):
        s, t = (torch.nonzero(m[p] >= 0)[:, 0] for m in (sm, tm))
        out = out.index_add(0, t[tm[p, t].argsort()], x[s[sm[p, s].argsort()]] @ w[order[p].long()])
    return out


@pytest.mark.parametrize("kernel,stride,transposed", [(3, 1, False), (2, 2, False), (2, 2, True), (5, 1, False)])
@pytest.mark.parametrize("dtype,bound", [(torch.float32, 1e-5), (torch.float16, 1e-2)])
@pytest.mark.parametrize("strided", [False, True])
def test_second_derivatives(kernel, stride, transposed, dtype, bound, strided):
    gen = torch.Generator(device=DEV).manual_seed(kernel + stride)
    i = torch.randperm(10 ** 3, generator=gen, device=DEV)[:400].sort().values
    coords = torch.stack([i // 100, i // 10 % 10, i % 10], 1).int()
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    make = lambda tr: minuet.nn.SparseConv(3, 8, 16, kernel, stride=stride, transposed=tr, dtype=dtype, device=DEV)
    conv, at, at_stride = make(False), coords, 1
    minuet.set_kernel_map_cache(conv, cache)
    if transposed:
        at, at_stride, _ = conv.prepare(coords, 1, None)
        conv = make(True)
        minuet.set_kernel_map_cache(conv, cache)
    x = torch.randn(len(at), 16, generator=gen, device=DEV).to(dtype)
    x = (x[:, ::2] if strided else x[:, :8].contiguous()).detach().requires_grad_()
    rows = len(conv.prepare(at, at_stride, None)[0])
    v = torch.randn(rows, 16, generator=gen, device=DEV).to(dtype)

    def second(out, inputs, v):
        wide = lambda t: t if t.dtype == torch.float64 else t.float()
        gx, gw = torch.autograd.grad((wide(out).square() * v).sum(), inputs, create_graph=True)
        return gx, gw, *torch.autograd.grad(wide(gx).square().sum(), inputs, retain_graph=True), \
            *torch.autograd.grad(wide(gw).square().sum() * 1e-2, inputs)

    with torch.no_grad():
        conv.kernel.mul_(0.5)
    tensor = minuet.SparseTensor(x, at, stride=at_stride)
    got = second(conv(tensor).F, (x, conv.kernel), v)
    maps = conv._lookup(tensor)[3:6]
    x64, w64 = x.detach().double().requires_grad_(), conv.kernel.detach().double().requires_grad_()
    want = second(_plain(x64, w64, *maps, rows), (x64, w64), v.double())
    for a, b in zip(got, want):
        assert float(((a.double() - b).norm() / b.norm()).detach()) < bound


def test_third_derivative():
    coords = torch.stack(torch.meshgrid(*3 * [torch.arange(4, device=DEV)], indexing="ij"), -1).view(-1, 3).int()
    conv, cache = minuet.nn.SparseConv3d(4, 4, 3, device=DEV), minuet.nn.KernelMapCache(3, torch.int32, DEV)
    minuet.set_kernel_map_cache(conv, cache)
    x = torch.randn(64, 4, device=DEV, requires_grad=True)

    def third(out, x, w):
        g, = torch.autograd.grad(out.pow(4).sum(), w, create_graph=True)
        h, = torch.autograd.grad(g.square().sum(), x, create_graph=True)
        return torch.autograd.grad(h.square().sum(), (x, w))

    tensor = minuet.SparseTensor(x, coords)
    got = third(conv(tensor).F, x, conv.kernel)
    x64, w64 = x.detach().double().requires_grad_(), conv.kernel.detach().double().requires_grad_()
    want = third(_plain(x64, w64, *conv._lookup(tensor)[3:6], 64), x64, w64)
    for a, b in zip(got, want):
        assert float((a.detach().double() - b).norm() / b.norm()) < 1e-4
