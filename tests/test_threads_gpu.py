"""Layers called from threads that have not used the GPU before, and from several at a time."""
import threading

import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _in_threads(count, call):
    results, errors = [None] * count, []

    def work(i):
        try:
            with torch.no_grad():
                results[i] = call()
        except Exception as error:           # noqa: BLE001 (shown by the assertion below)
            errors.append(error)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    return results


@pytest.mark.parametrize("dtype,algorithm", [(torch.float32, "auto"), (torch.float16, "implicit"),
                                             (torch.float16, "explicit")])
@pytest.mark.parametrize("warm", [False, True])
def test_layers_in_new_threads(dtype, algorithm, warm):
    coords = torch.stack(torch.meshgrid(*3 * [torch.arange(12, device=DEV)], indexing="ij"), -1).view(-1, 3).int()
    conv = minuet.nn.SparseConv3d(32, 32, 3, dtype=dtype, device=DEV)
    cache = minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)
    minuet.set_kernel_map_cache(conv, cache)
    conv.tunable_config.update(algorithm=algorithm)
    x = minuet.SparseTensor(torch.randn(len(coords), 32, device=DEV).to(dtype), coords)
    want = conv(x).F
    if not warm:
        cache.reset()
        conv.prepare(coords, 1, None)        # the map, without its tables
    torch.cuda.synchronize()
    for got in _in_threads(4, lambda: [conv(x).F for _ in range(10)]):
        assert all(torch.equal(g, want) for g in got)


def test_dense_products_in_new_threads():
    x, w = torch.randn(300, 32, device=DEV).half(), torch.randn(32, 64, device=DEV).half()
    w_t = F.transpose_weights(w)
    want = F.dense_forward(x, w)
    torch.cuda.synchronize()
    for got in _in_threads(3, lambda: F.dense_forward(x, w, weights_t=w_t)):
        assert torch.equal(got, want)
