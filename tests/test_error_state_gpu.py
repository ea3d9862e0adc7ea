"""The host path's looks at events leave the CUDA errors of other calls alone."""
import ctypes

import pytest
import torch

from minuet_b200 import _lib, engine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INVALID_DEVICE = 101


def test_a_pending_error_of_another_call_is_kept():
    runtime = ctypes.CDLL("libcudart.so.12")          # the one that torch has loaded
    coords = torch.stack(torch.meshgrid(*3 * [torch.arange(8, device=DEV)], indexing="ij"), -1).view(-1, 3).int()
    engine.poll_status(DEV)
    torch.cuda._sleep(20_000_000)
    for _ in range(3):                                # copies that have not landed, and then some that have
        engine.poll_status(DEV)
    layout = _lib.host().root_keys(coords, None, 1, 64)[0]
    assert layout.margin == 64
    for wait in (False, True):
        if wait:
            torch.cuda.synchronize()
        assert runtime.cudaSetDevice(999) == INVALID_DEVICE
        try:
            engine.poll_status(DEV)
            assert runtime.cudaPeekAtLastError() == INVALID_DEVICE
        finally:
            runtime.cudaGetLastError()
    torch.cuda.synchronize()
