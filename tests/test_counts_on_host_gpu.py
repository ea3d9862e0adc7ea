"""The counts that the host reads: of a strided level and a voxelisation (row counts and cloud starts, written to
host memory by the kernel where they fit the buffer (1024 values: 1020 clouds), copied beyond) and of kernel
maps, several of them on their way at once and inside stream captures."""
import numpy as np
import pytest
import torch

import minuet_b200 as minuet
from minuet_b200 import engine
from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("clouds", [1, 2, 1019, 1020, 1021, 1500])
def test_counts_and_cloud_starts(clouds):
    rng = np.random.default_rng(clouds)
    per_cloud = [np.unique(rng.integers(-9, 9, (int(rng.integers(1, 40)), 3)), axis=0) for _ in range(clouds)]
    starts = np.cumsum([0] + [len(c) for c in per_cloud])
    coords = torch.as_tensor(np.concatenate(per_cloud), dtype=torch.int32, device=DEV)
    bounds = torch.as_tensor(starts, device=DEV) if clouds > 1 else None
    want = [np.unique(c // 2 * 2, axis=0) for c in per_cloud]
    want_starts = np.cumsum([0] + [len(c) for c in want])
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    out, stride, out_bounds = cache.get_target_coordinates(coords, bounds, 1, 2)
    assert stride == (2, 2, 2) and np.array_equal(out.cpu().numpy(), np.concatenate(want))
    if clouds > 1:
        assert np.array_equal(out_bounds.cpu().numpy(), want_starts)
    sizes = cache.get_kernel_map(coords, 1, bounds, out, stride, out_bounds, 2, 1)[3]
    assert int(sizes.sum()) == len(coords)                    # every voxel has one parent
    # the same counts from points, the means on the way when the host goes on
    points = coords.float() + 0.5
    features = torch.rand(len(coords), 5, device=DEV)
    result = F.voxelize(points, 2.0, batch_dims=bounds, features=features, return_inverse=True)
    voxels, inverse, means = result[0], result[-2], result[-1]
    assert np.array_equal(voxels.cpu().numpy() * 2, np.concatenate(want))
    ref = torch.zeros(len(voxels), 5, device=DEV, dtype=torch.float64).index_add_(0, inverse, features.double())
    ref /= torch.bincount(inverse, minlength=len(voxels))[:, None]
    assert float((means - ref).abs().max()) < 8 * 2.0 ** -23   # at most eight values below one


def _map_of(coords, kernel):
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    return cache, cache.get_kernel_map(coords, 1, None, coords, 1, None, kernel, 1)


def test_many_counts_on_their_way_at_once():
    """Buffers of maps that are gone before the GPU has written them are not handed out again too early."""
    rng = np.random.default_rng(0)
    clouds = [torch.as_tensor(np.unique(rng.integers(0, 30, (200 * (k + 1), 3)), axis=0), dtype=torch.int32, device=DEV)
              for k in range(24)]
    for _ in range(2):                                # (the second time with buffers that were given back)
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)                 # some 10 ms in front of the maps
        kept = []
        for k, c in enumerate(clouds):
            cache, result = _map_of(c, 3 if k % 3 else 2)
            if k % 2:
                kept.append((cache, result))
            del cache, result
        for _, (_, tm, _, sizes) in kept:
            assert engine.host_copy(sizes).tolist() == (tm >= 0).sum(1).tolist()


@pytest.mark.parametrize("kernel", [3, 5])            # 27 offsets, and more than the fused build takes
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_a_map_built_inside_a_capture(kernel, mode):
    rng = np.random.default_rng(kernel)
    first, second = (torch.as_tensor(np.unique(rng.integers(0, 20, (4000, 3)), axis=0)[:2500], dtype=torch.int32,
                                     device=DEV) for _ in range(2))
    coords = first.clone()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _map_of(coords, kernel)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        cache, (sm, tm, order, sizes) = _map_of(coords, kernel)
    for points in (first, second):
        coords.copy_(points)
        graph.replay()
        want = _map_of(points.clone(), kernel)[1]
        for got, expected in zip((sm, tm, order, sizes), want):
            assert torch.equal(got, expected)
    # what every replay writes anew is not read as if it were fixed, and nothing is left behind
    conv = minuet.nn.SparseConv3d(4, 4, kernel, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    with pytest.raises(RuntimeError, match="stream capture"):
        conv(minuet.SparseTensor(torch.ones(len(coords), 4, device=DEV), coords))
    del conv, cache, sm, tm, order, sizes, graph
    for _ in range(3):
        _, (_, tm, _, sizes) = _map_of(first, kernel)
        assert engine.host_copy(sizes).tolist() == (tm >= 0).sum(1).tolist()


def test_a_stream_that_is_first_used_inside_captures():
    """Two graphs captured on one new stream, the second replayed first, then work outside a capture there."""
    coords = [torch.as_tensor(np.unique(np.random.default_rng(k).integers(0, 20, (4000, 3)), axis=0), dtype=torch.int32,
                              device=DEV) for k in range(2)]
    want = [_map_of(c, 3)[1] for c in coords]
    stream, graphs, maps = torch.cuda.Stream(), [], []
    for c in coords:
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=stream):
            maps.append(_map_of(c, 3))
    for k in (1, 1, 0, 1):
        for t in maps[k][1]:
            t.fill_(-7)
        graphs[k].replay()
        assert all(torch.equal(got, expected) for got, expected in zip(maps[k][1], want[k]))
    del graphs, maps
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        got = _map_of(coords[0], 3)[1]
        assert engine.host_copy(got[3]).tolist() == engine.host_copy(want[0][3]).tolist()
        assert all(torch.equal(a, b) for a, b in zip(got, want[0]))
