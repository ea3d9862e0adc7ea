"""What is derived from a kernel map once (tables, lists, counts) follows the map: masks that are written
to, or come with other pair counts, give the results of what they hold now."""
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import engine
from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(dtype, rows=2500, channels=32):
    gen = torch.Generator(device=DEV).manual_seed(rows)
    i = torch.randperm(20 ** 3, generator=gen, device=DEV)[:rows].sort().values
    coords = torch.stack([i // 400, i // 20 % 20, i % 20], 1).int()
    conv = minuet.nn.SparseConv3d(channels, channels, 3, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.kernel.data.copy_(torch.randint(-1, 2, conv.kernel.shape, generator=gen, device=DEV))
    x = torch.randint(-1, 2, (rows, channels), generator=gen, device=DEV).to(dtype)
    return conv, cache, x, coords, cache.get_kernel_map(coords, 1, None, coords, 1, None, 3, 1)


def _sums(x, w, sm, tm, order):
    """The convolution that the masks describe, in whole numbers."""
    out = torch.zeros(len(x), w.shape[2], device=DEV)
    for p in range(len(sm)):
        s, t = (torch.nonzero(m[p] >= 0)[:, 0] for m in (sm, tm))
        out[t[tm[p, t].argsort()]] += x[s[sm[p, s].argsort()]].float() @ w[order[p].long()].float()
    return out


def _drop_last_pair(sm, tm, sizes, p):
    last = int(sizes[p]) - 1
    sm[p][sm[p] == last] = -1
    tm[p][tm[p] == last] = -1
    sizes[p] = last


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("algorithm", ["auto", "explicit", "implicit"])
@pytest.mark.parametrize("own", [True, False])
def test_masks_written_between_calls(dtype, algorithm, own):
    conv, cache, x, coords, (sm, tm, order, sizes) = _layer(dtype)
    if not own:
        sm, tm, order, sizes = (t.clone() for t in (sm, tm, order, sizes))
    call = lambda: F.sparse_convolution_forward(x, conv.kernel, sm, tm, order, sizes, 1, 1, algorithm=algorithm)
    for _ in range(2):
        assert torch.equal(call().float(), _sums(x, conv.kernel, sm, tm, order))
        assert torch.equal(call().float(), _sums(x, conv.kernel, sm, tm, order))
        if own:                                      # the layer that has this map in its cache
            conv.tunable_config.update(algorithm=algorithm)
            assert torch.equal(conv(minuet.SparseTensor(x, coords)).F.float(), _sums(x, conv.kernel, sm, tm, order))
        _drop_last_pair(sm, tm, sizes, 0)
        _drop_last_pair(sm, tm, sizes, 5)
    assert torch.equal(call().float(), _sums(x, conv.kernel, sm, tm, order))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_the_same_masks_with_other_counts(dtype):
    """An offset without pairs whose count the caller keeps in another tensor, and host values."""
    conv, cache, x, coords, (sm, tm, order, sizes) = _layer(dtype)
    sm, tm = sm.clone(), tm.clone()
    call = lambda n: F.sparse_convolution_forward(x, conv.kernel, sm, tm, order, n, 1, 1)
    assert torch.equal(call(sizes).float(), _sums(x, conv.kernel, sm, tm, order))
    sm[0] = -1
    tm[0] = -1
    other = torch.cat([sizes[:1] * 0, sizes[1:]])
    for n in (other, other.cpu(), other.long()):
        assert torch.equal(call(n).float(), _sums(x, conv.kernel, sm, tm, order))


@pytest.mark.needs_grad
def test_a_map_written_before_the_backward_pass_is_an_error():
    conv, cache, x, coords, (sm, tm, order, sizes) = _layer(torch.float32)
    out = conv(minuet.SparseTensor(x.requires_grad_(), coords)).F
    sm[0] = -1
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        out.sum().backward()


def test_unwritten_maps_keep_their_plan():
    conv, cache, x, coords, (sm, tm, order, sizes) = _layer(torch.float16)
    plan, swapped = engine.plan_of(sm, tm, sizes)
    assert engine.plan_of(sm, tm, sizes)[0] is plan and not swapped
    assert engine.plan_of(sm, tm, engine.host_copy(sizes))[0] is plan
    assert engine.plan_of(tm, sm, sizes) == (plan, True)
    a, b = sm.clone(), tm.clone()
    other = engine.plan_of(a, b, sizes)[0]
    assert other is not plan and engine.plan_of(a, b, sizes)[0] is other


@pytest.mark.needs_grad
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_ranks_without_a_partner_make_no_pair(dtype):
    """A caller's own masks that do not fit together: entries that one side lacks, or that the counts
    have no place for, are no pairs, and nothing is read through them."""
    conv, cache, x, coords, (sm, tm, order, sizes) = _layer(dtype)
    want_s, want_t, a, b = sm.clone(), tm.clone(), sm.clone(), tm.clone()
    b[3][b[3] == 2] = -1                       # only the source side has rank 2 of row 3
    want_s[3][sm[3] == 2] = want_t[3][tm[3] == 2] = -1
    a[4][a[4] == 7] = -1                       # only the target side has rank 7 of row 4
    want_s[4][sm[4] == 7] = want_t[4][tm[4] == 7] = -1
    free_s, free_t = (int((m[26] >= 0).logical_and(m[5] < 0).nonzero()[0]) for m in (sm, tm))
    a[5, free_s] = b[5, free_t] = 1 << 30      # far behind the row's last rank
    sums = torch.zeros(len(x), 32, device=DEV)
    for p in range(27):
        rank = torch.full((len(x),), -1, device=DEV)
        s = torch.nonzero(want_s[p] >= 0)[:, 0]
        rank[want_s[p, s].long()] = s
        t = torch.nonzero(want_t[p] >= 0)[:, 0]
        sums[t] += x[rank[want_t[p, t].long()]].float() @ conv.kernel[order[p].long()].detach().float()
    x.requires_grad_()
    out = F.sparse_convolution_forward(x, conv.kernel, a, b, order, sizes, 1, 1, algorithm="implicit")
    gx, gw = torch.autograd.grad(out, (x, conv.kernel), torch.ones_like(out))
    assert torch.equal(out.float(), sums)
    assert bool(torch.isfinite(gx).all()) and bool(torch.isfinite(gw).all())
    torch.cuda.synchronize()
