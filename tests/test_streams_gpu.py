"""What a kernel map's plan makes on first use (neighbour tables, pair lists) on several streams and inside
stream captures."""
import pytest
import torch

import minuet_b200 as minuet

pytestmark = [pytest.mark.gpu, pytest.mark.needs_grad]
DEV = "cuda:0"


def _layer(dtype, algorithm):
    gen = torch.Generator(device=DEV).manual_seed(1)
    i = torch.randperm(40 ** 3, generator=gen, device=DEV)[:20_000].sort().values
    coords = torch.stack([i // 1600, i // 40 % 40, i % 40], 1).int()
    conv = minuet.nn.SparseConv3d(32, 32, 3, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm=algorithm)
    conv.prepare(coords, 1, None)
    x = torch.randn(len(coords), 32, generator=gen, device=DEV).to(dtype).requires_grad_()
    return conv, cache, x, coords


def _step(conv, x, coords):
    out = conv(minuet.SparseTensor(x, coords)).F
    return (out.detach(), *torch.autograd.grad(out, (x, conv.kernel), torch.ones_like(out)))


@pytest.mark.parametrize("dtype,algorithm", [(torch.float32, "auto"), (torch.float16, "implicit"),
                                             (torch.float16, "explicit")])
def test_the_first_use_on_one_stream_and_the_second_on_another(dtype, algorithm):
    conv, cache, x, coords = _layer(dtype, algorithm)
    want = _step(conv, x, coords)
    for _ in range(5):
        cache.reset()
        conv.prepare(coords, 1, None)
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in range(3)]
        got = []
        for k, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                if k == 0:
                    torch.cuda._sleep(20_000_000)      # some 10 ms in front of the tables
                got.append(_step(conv, x, coords))
        torch.cuda.synchronize()
        for result in got:
            assert all(torch.equal(a, b) for a, b in zip(result, want))


@pytest.mark.parametrize("dtype,algorithm", [(torch.float32, "auto"), (torch.float16, "implicit"),
                                             (torch.float16, "explicit")])
def test_tables_first_needed_inside_a_capture(dtype, algorithm):
    conv, cache, x, coords = _layer(dtype, algorithm)
    want = _step(conv, x, coords)
    cache.reset()
    with torch.no_grad():
        conv(minuet.SparseTensor(x, coords))           # the backward pass' tables are still missing
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = _step(conv, x, coords)
    eager = _step(conv, x, coords)                     # before any replay has run
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(eager, want))
    for _ in range(2):
        for t in captured:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(captured, want))
