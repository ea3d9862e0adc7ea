"""Layers, networks and caches that have run are copied and saved like any other module, and follow their
attributes."""
import copy
import io
import pickle

import pytest
import torch

import minuet_b200 as minuet
from minuet_b200.unet import SparseUNet

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cache():
    return minuet.nn.KernelMapCache(ndim=3, dtype=torch.int32, device=DEV)


def _input(dtype, channels=8, rows=900):
    gen = torch.Generator(device=DEV).manual_seed(rows)
    i = torch.randperm(14 ** 3, generator=gen, device=DEV)[:rows].sort().values
    coords = torch.stack([i // 196, i // 14 % 14, i % 14], 1).int()
    return minuet.SparseTensor(torch.randn(rows, channels, generator=gen, device=DEV).to(dtype), coords)


def _through_a_file(module):
    file = io.BytesIO()
    torch.save(module, file)
    file.seek(0)
    return torch.load(file, weights_only=False)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("copying", [copy.deepcopy, _through_a_file, lambda m: pickle.loads(pickle.dumps(m))])
@pytest.mark.parametrize("cache", ["none", "reset"])
def test_a_layer_that_has_run(dtype, copying, cache):
    x, conv, maps = _input(dtype), minuet.nn.SparseConv3d(8, 8, 3, dtype=dtype, device=DEV), _cache()
    minuet.set_kernel_map_cache(conv, maps)
    want = conv(x).F
    conv.forward_fused(x, relu=True)
    maps.reset()
    if cache == "none":
        conv.set_kernel_map_cache(None)
    twin = copying(conv)
    if cache == "none":
        twin.set_kernel_map_cache(_cache())
    assert twin._kernel_map_cache is not maps
    assert torch.equal(twin(x).F, want)
    conv.set_kernel_map_cache(maps)
    assert torch.equal(conv(x).F, want)          # the original goes on


def test_a_network_that_has_run():
    net, maps, x = SparseUNet(4, num_classes=5, channels=(8, 16, 32, 64), stem_channels=8).to(DEV).eval(), _cache(), _input(
        torch.float32, 4)
    minuet.set_kernel_map_cache(net, maps)
    want = net(x).F
    maps.reset()
    assert torch.equal(copy.deepcopy(net)(x).F, want)


def test_a_cache_in_use_is_not_copied():
    conv, maps, x = minuet.nn.SparseConv3d(8, 8, 3, device=DEV), _cache(), _input(torch.float32)
    minuet.set_kernel_map_cache(conv, maps)
    conv(x)
    for copying in (copy.deepcopy, pickle.dumps):
        with pytest.raises(ValueError, match="reset"):
            copying(maps)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_a_layer_whose_geometry_is_changed(dtype):
    """What a layer looks up follows its attributes, not those it was made with."""
    x = _input(dtype)
    conv = minuet.nn.SparseConv3d(8, 8, 3, dtype=dtype, device=DEV)
    minuet.set_kernel_map_cache(conv, _cache())
    conv(x)
    for size, stride, dilation in (((2, 2, 2), (1, 1, 1), (1, 1, 1)), ((3, 1, 1), (1, 1, 1), (2, 1, 1)),
                                   ((2, 2, 2), (2, 2, 2), (1, 1, 1)), ((1, 1, 1), (1, 1, 1), (1, 1, 1))):
        made = minuet.nn.SparseConv3d(8, 8, size, stride=stride, dilation=dilation, dtype=dtype, device=DEV)
        minuet.set_kernel_map_cache(made, _cache())
        conv.kernel_size, conv.stride, conv.dilation, conv.kernel = size, stride, dilation, made.kernel
        want, got = made(x), conv(x)
        assert torch.equal(got.F, want.F) and torch.equal(got.C, want.C) and got.stride == want.stride
