"""1x1x1 convolutions in training: the weight's gradient where it is a kernel of this library against fp64 and, to the
bit, where the values are small whole numbers; and everything else that autograd does with the layer, against the
plain product."""
import pytest
import torch
from torch.autograd import forward_ad

import minuet_b200 as minuet
from minuet_b200 import _lib

pytestmark = [pytest.mark.gpu, pytest.mark.needs_grad]
DEV = "cuda:0"


def _layer(c_in, c_out, dtype=torch.float32):
    conv = minuet.nn.SparseConv3d(c_in, c_out, 1, bias=False, device=DEV, dtype=dtype)
    return conv, lambda x: conv(minuet.SparseTensor(x, torch.zeros(len(x), 3, dtype=torch.int32, device=DEV))).F


def _matrix(conv):
    return conv.kernel.view(conv.in_channels, conv.out_channels)


def _own(out):
    return "DenseProduct" in out.grad_fn.name()


@pytest.mark.parametrize("c_in,c_out", [(1, 1), (32, 13), (33, 32), (36, 100), (64, 64), (65, 20), (128, 256), (256, 256)])
@pytest.mark.parametrize("rows", [1024, 1025, 1151, 4097, 131_072, 131_073])
def test_gradients(rows, c_in, c_out):
    gen = torch.Generator(device=DEV).manual_seed(rows + c_in)
    conv, run = _layer(c_in, c_out)
    x = torch.randn(rows, c_in, generator=gen, device=DEV).requires_grad_()
    g = torch.randn(rows, c_out, generator=gen, device=DEV)
    out = run(x)
    assert _own(out) == (c_in * c_out <= 1 << 15 or rows <= 1 << 17)
    plain = x @ _matrix(conv)
    assert torch.equal(out, plain)
    gx, gw = torch.autograd.grad(out, (x, conv.kernel), g)
    assert torch.equal(gx, torch.autograd.grad(plain, x, g)[0])
    a, b = x.detach().double(), g.double()
    # `rows` products and their sums in fp32, in any order
    bound = (rows + 1) * 2.0 ** -24 * (a.abs().t() @ b.abs())
    assert bool(((gw.view(c_in, c_out).double() - a.t() @ b).abs() <= bound).all())
    whole = [torch.randint(-3, 4, t.shape, generator=gen, device=DEV).float() for t in (x, g)]
    gw, = torch.autograd.grad(run(whole[0]), conv.kernel, whole[1])    # sums below 9 * 131 073 < 2^24: exact
    assert torch.equal(gw.view(c_in, c_out), (whole[0].double().t() @ whole[1].double()).float())


@pytest.mark.parametrize("rows,c_in,c_out,tf32", [
    (4097, 1, 48, False), (4097, 96, 1, False), (16_383, 7, 64, False), (2047, 33, 36, False), (400_000, 13, 40, False),
    (131_072, 4, 4096, False), (20_000, 192, 128, True), (8191, 64, 64, True), (500_000, 64, 80, True)])
def test_weight_gradients_that_are_left_to_torch(rows, c_in, c_out, tf32):
    """One channel, channels not in fours into many, many tiles, a faster GEMM that the caller allows: its bits."""
    gen = torch.Generator(device=DEV).manual_seed(rows + c_in)
    conv, run = _layer(c_in, c_out)
    x, g = (torch.randn(rows, c, generator=gen, device=DEV) for c in (c_in, c_out))
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = tf32
    try:
        got, want = (torch.autograd.grad(out, conv.kernel, g)[0] for out in (run(x), x @ _matrix(conv)))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before
    assert torch.equal(got, want)


@pytest.mark.parametrize("rows,c_in,c_out", [(1024, 32, 20), (8192, 64, 64), (8192, 128, 64)])
def test_weight_gradients_in_fp32_where_tf32_is_allowed(rows, c_in, c_out):
    gen = torch.Generator(device=DEV).manual_seed(rows + c_in)
    conv, run = _layer(c_in, c_out)
    x, g = (torch.randn(rows, c, generator=gen, device=DEV) for c in (c_in, c_out))
    want, = torch.autograd.grad(run(x), conv.kernel, g)
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        got, = torch.autograd.grad(run(x), conv.kernel, g)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before
    assert torch.equal(got, want)


@pytest.mark.parametrize("case", ["few rows", "half", "strided", "frozen", "autocast", "wide", "no rows", "function mode"])
def test_calls_that_stay_a_plain_product(case):
    gen = torch.Generator(device=DEV).manual_seed(1)
    c_in, c_out = (512, 512) if case == "wide" else (32, 24)
    conv, run = _layer(c_in, c_out, torch.float16 if case == "half" else torch.float32)
    x = torch.randn({"few rows": 1023, "no rows": 0}.get(case, 2000), c_in, generator=gen, device=DEV)
    if case == "half":
        x = x.half()
    if case == "strided":
        x = torch.randn(2000, 2 * c_in, generator=gen, device=DEV)[:, ::2]
    if case == "frozen":
        conv.kernel.requires_grad_(False)
    x.requires_grad_()
    if case == "autocast":
        with torch.autocast("cuda", torch.float16):
            out, want = run(x), x @ _matrix(conv)
    elif case == "function mode":
        with torch.device("cuda:0"):
            out, want = run(x), x @ _matrix(conv)
    else:
        out, want = run(x), x @ _matrix(conv)
    assert not _own(out) and out.dtype == want.dtype and torch.equal(out, want)


def test_transforms_of_the_layer():
    gen = torch.Generator(device=DEV).manual_seed(2)
    conv, run = _layer(32, 24)
    w = conv.kernel
    x, g, v = (torch.randn(2000, c, generator=gen, device=DEV) for c in (32, 24, 32))

    def plain(a, kernel):
        return a @ kernel.view(32, 24)

    def layer(a, kernel):
        return torch.func.functional_call(conv, {"kernel": kernel}, (minuet.SparseTensor(a, torch.zeros(
            2000, 3, dtype=torch.int32, device=DEV)),)).F

    for f in (torch.func.grad(lambda f, a, k: (f(a, k) * g).sum(), argnums=(1, 2)),
              lambda f, a, k: torch.func.vmap(lambda b: f(b, k))(torch.stack([a, v]))):
        for got, want in zip(f(layer, x, w), f(plain, x, w)):
            torch.testing.assert_close(got, want, rtol=0, atol=0)
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(x, v)
        for got, want in zip(forward_ad.unpack_dual(layer(dual, w)), forward_ad.unpack_dual(plain(dual, w))):
            assert torch.equal(got, want)

    # the backward pass under a transform, of a forward pass under none
    a = x.clone().requires_grad_()
    out, ref = run(a), plain(a, w)
    assert _own(out)
    gs = torch.stack([g, 2 * g])
    for got, want in zip(*(torch.autograd.grad(o, (a, w), gs, is_grads_batched=True, retain_graph=True) for o in (out, ref))):
        assert torch.equal(got, want)
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(g, 2 * g)
        got, want = (forward_ad.unpack_dual(torch.autograd.grad(o, w, dual, retain_graph=True)[0]) for o in (out, ref))
        assert torch.equal(got.primal, want.primal) and torch.equal(got.tangent, want.tangent)


def test_second_derivatives_hooks_layouts_streams_and_capture():
    gen = torch.Generator(device=DEV).manual_seed(3)
    conv, run = _layer(32, 24)
    w = conv.kernel
    x, g, v = (torch.randn(2000, c, generator=gen, device=DEV) for c in (32, 24, 32))
    x.requires_grad_()

    def second(out):
        h = g.clone().requires_grad_()
        gx, gw = torch.autograd.grad(out, (x, w), h, create_graph=True)
        return torch.autograd.grad((gx * v).sum() + (gw ** 2).sum(), (x, w, h))

    for got, want in zip(second(run(x)), second(x @ _matrix(conv))):
        assert torch.equal(got, want)

    want = torch.autograd.grad(run(x), (x, w), g)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(DEV)):
        out = run(x)
    assert all(map(torch.equal, torch.autograd.grad(out, (x, w), g), want))
    assert all(map(torch.equal, torch.autograd.grad(run(x), (x, w), g.t().contiguous().t()), want))
    same = torch.autograd.grad(run(x), w, g[:1].expand(2000, 24))[0]
    assert torch.equal(same, torch.autograd.grad(run(x), w, g[:1].repeat(2000, 1))[0])
    # rows off a 16-byte boundary
    off = torch.randn(2000 * 32 + 1, generator=gen, device=DEV)[1:].view(2000, 32)
    torch.testing.assert_close(torch.autograd.grad(run(off), w, g)[0], torch.autograd.grad(run(off.clone()), w, g)[0])

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):     # (leaves of its own: a leaf's gradient belongs to the stream it was first used on)
        conv2, run2 = _layer(32, 24)
        conv2.load_state_dict(conv.state_dict())
        x2 = x.detach().clone().requires_grad_()
        got = torch.autograd.grad(run2(x2), (x2, conv2.kernel), g)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            captured = torch.autograd.grad(run2(x2), (x2, conv2.kernel), g)
        graph.replay()
    torch.cuda.current_stream().wait_stream(side)
    assert all(map(torch.equal, got, want)) and all(map(torch.equal, captured, want))
    out = run(x)
    x.detach().add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        torch.autograd.grad(out, w, g)


def test_values_that_are_not_finite():
    conv, run = _layer(8, 8)
    x = torch.ones(3000, 8, device=DEV)
    x[2999, 3], x[17, 5] = float("inf"), float("nan")
    gw, = torch.autograd.grad(run(x), conv.kernel, torch.ones(3000, 8, device=DEV))
    gw = gw.view(8, 8)
    assert bool(gw[3].isinf().all()) and bool(gw[5].isnan().all()) and bool((gw[[0, 1, 2, 4, 6, 7]] == 3000).all())
