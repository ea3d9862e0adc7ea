"""The sort's bounded look-back: a wait that runs out is reported, and what the sort leaves behind can
still be used as indices."""
import pytest
import torch

from minuet_b200 import _lib, engine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _sort(keys, bits, wait_limit):
    lib, n = _lib.load(), len(keys)
    index = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ws = torch.full((lib.mn_map_workspace_bytes(n, n, 1),), 0xff, dtype=torch.uint8, device=DEV)
    _lib.check(lib.mn_arg_sort_keys(engine.ptr(keys), n, bits, wait_limit, engine.ptr(index), engine.ptr(status),
                                    engine.ptr(ws), ws.numel(), engine.stream_ptr(torch.device(DEV))), "arg_sort_keys")
    return index, int(status)


@pytest.mark.parametrize("n,bits", [(1, 1), (1025, 9), (300_000, 20), (700_001, 44)])
def test_indices_stay_in_range_when_the_wait_runs_out(n, bits):
    gen = torch.Generator(device=DEV).manual_seed(n)
    keys = torch.randint(0, 1 << bits, (n,), generator=gen, device=DEV)
    want = torch.sort(keys, stable=True).indices
    index, status = _sort(keys, bits, 0)
    assert status == 0 and torch.equal(index, want)
    ran_out = 0
    for _ in range(20):
        index, status = _sort(keys, bits, 1)
        assert status in (0, engine.STATUS_GRID_TIMEOUT)
        assert int(index.min()) >= 0 and int(index.max()) < n
        assert status != 0 or torch.equal(index, want)
        ran_out += status != 0
    assert n < 100_000 or ran_out > 0
