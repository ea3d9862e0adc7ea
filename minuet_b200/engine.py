"""Torch-facing glue over the C ABI: pointers, streams, workspaces, key specs.

PyTorch is used here only for device memory, the current stream and the final
device-to-host reads.  All compute is in ``libminuet_b200.so``.
"""
import ctypes
import weakref
from typing import Optional, Sequence

import numpy as np
import torch

from minuet_b200 import _lib
from minuet_b200._lib import KeySpec

DEFAULT_MARGIN = 64
# When set to a list, every convolution appends a dict with its shape (S, T, O, E,
# c_in, c_out, algorithm); benchmarks use it to compute per-layer rooflines.
LAYER_LOG = None
_DTYPE_CODE = {torch.float32: _lib.MN_F32, torch.float16: _lib.MN_F16,
               torch.bfloat16: _lib.MN_BF16}


def event_pair_begin(device):
    """Two timing events, the first recorded now on the current stream (per-layer
    times for LAYER_LOG)."""
    pair = (torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
    pair[0].record(torch.cuda.current_stream(device))
    return pair


def event_pair_end(pair, device):
    pair[1].record(torch.cuda.current_stream(device))


def lib():
    return _lib.load()


def require_cuda(*tensors):
    """The reference raises NotImplementedError for non-CUDA tensors
    (minuet/nn/functional/indexing.py:56,127); so does this engine."""
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise NotImplementedError("minuet_b200 runs on CUDA tensors only (no CPU path)")


def ptr(t: Optional[torch.Tensor]):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def np_ptr(a: Optional[np.ndarray]):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def _device_index(device) -> int:
    if isinstance(device, int):
        return device
    if not isinstance(device, torch.device):
        device = torch.device(device)
    return torch.cuda.current_device() if device.index is None else device.index


def raw_stream(device) -> int:
    """The current stream of ``device`` as an integer handle (the raw query costs a
    fraction of a microsecond; building a ``torch.cuda.Stream`` object costs several, and
    the map step asks for the stream a dozen times per build)."""
    return torch._C._cuda_getCurrentRawStream(_device_index(device))


def stream_ptr(device) -> ctypes.c_void_p:
    return ctypes.c_void_p(raw_stream(device))


def dtype_code(dtype: torch.dtype) -> int:
    if dtype not in _DTYPE_CODE:
        raise RuntimeError(f"Cannot find implementation of sparse convolution for {dtype}")
    return _DTYPE_CODE[dtype]


_WORKSPACE_CACHE_BYTES = 64 << 20
_workspaces = {}


def workspace(nbytes: int, device) -> torch.Tensor:
    """Scratch bytes for one library call.  Requests up to 64 MiB share one grow-only
    buffer per (device, stream): calls on one stream run in order, so the next call may
    overwrite what the previous one left.  Larger requests get a buffer of their own."""
    nbytes = max(int(nbytes), 256)
    if nbytes > _WORKSPACE_CACHE_BYTES:
        return torch.empty(nbytes, dtype=torch.uint8, device=device)
    key = (_device_index(device), raw_stream(device))
    buf = _workspaces.get(key)
    if buf is None or buf.numel() < nbytes:
        buf = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8,
                          device=torch.device("cuda", key[0]))
        _workspaces[key] = buf
    return buf


def as_i32_coords(coords: torch.Tensor) -> torch.Tensor:
    """The kernels read int32 coordinates; int64 tensors are narrowed (their
    values must fit, as the reference's subtraction-based comparisons already
    require |c| < 2**30, csrc/minuet/common/functions.h:94-105)."""
    if coords.dtype == torch.int32:
        return coords.contiguous()
    if coords.dtype == torch.int64:
        return coords.to(torch.int32).contiguous()
    raise ValueError(f"The coordinates tensor must be int32 or int64 but found {coords.dtype}")


def as_i64(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    if t is None:
        return None
    return t.to(torch.int64).contiguous()


# ---------------------------------------------------------------------------
# device status word
#   bit 1 (value 2): a coordinate fell outside the box the keys were built for
#   bit 2 (value 4): a bounded wait inside a tensor-core kernel ran out; the
#                    features that kernel wrote are invalid
#   bit 3 (value 8): the bounding box needs more than 63 key bits
# ---------------------------------------------------------------------------
STATUS_KEY_BOX = 2
STATUS_TC_TIMEOUT = 4
STATUS_KEY_BITS = 8
STATUS_GRID_TIMEOUT = 16


def control_block(device) -> torch.Tensor:
    """The ``MN_CTRL_WORDS`` int32 control block of (device, current stream): word 0
    is the status word, the rest is grid-barrier state of the cooperative kernels.
    One block per stream, because kernels of different streams may overlap."""
    return _lib.host().control_block(_device_index(device))


def status_word(device) -> torch.Tensor:
    """One-element view of the status word (the start of the control block)."""
    return control_block(device)[:1]


def decode_status(value: int) -> Optional[Exception]:
    """The exception a non-zero status word stands for (None for 0)."""
    value = int(value)
    if value == 0:
        return None
    parts = []
    if value & STATUS_TC_TIMEOUT:
        parts.append("a tensor-core kernel gave up waiting on one of its barriers: the "
                     "features it wrote are invalid (MN_ERR_DEVICE)")
    if value & STATUS_KEY_BITS:
        parts.append("the bounding box of the coordinates needs more than 63 key bits")
    if value & STATUS_KEY_BOX:
        parts.append("a coordinate lies outside the bounding box the sort/search keys were "
                     "built for (call KernelMapCache.reset() before feeding unrelated "
                     "coordinates)")
    if value & STATUS_GRID_TIMEOUT:
        parts.append("a grid-wide barrier of a cooperative kernel timed out: its outputs are "
                     "invalid (MN_ERR_DEVICE)")
    if value & ~(STATUS_KEY_BOX | STATUS_TC_TIMEOUT | STATUS_KEY_BITS | STATUS_GRID_TIMEOUT):
        parts.append(f"unknown device status bits 0x{value:x}")
    if value & STATUS_KEY_BITS and not value & (STATUS_TC_TIMEOUT | STATUS_GRID_TIMEOUT):
        return NotImplementedError("; ".join(parts))
    return RuntimeError("; ".join(parts))


def raise_on_status(value: int, device):
    error = decode_status(value)
    if error is not None:
        control_block(device).zero_()      # also resets the barrier state after a timeout
        raise error


def check_status(device):
    """Blocking read of the status word."""
    raise_on_status(int(status_word(device).item()), device)


def poll_status(device):
    """Non-blocking check for the forward path: queues an asynchronous copy of the
    status word into pinned memory and raises for any earlier copy that has
    landed with a non-zero value.  An error therefore surfaces at the latest one
    call after the kernel that raised it, without a host-device synchronisation."""
    raise_on_status(_lib.host().poll_status(_device_index(device)), device)


# ---------------------------------------------------------------------------
# key specs and keys
# ---------------------------------------------------------------------------

def make_keyspec(coord_tensors: Sequence[torch.Tensor], ndim: int, num_clouds: int,
                 margin: int) -> KeySpec:
    """Bounding box on the device, one small D2H read, layout on the host."""
    tensors = [t for t in coord_tensors if t is not None and t.shape[0] > 0]
    spec = KeySpec()
    if not tensors:
        mm = np.array([0, 0, 0, 0, 0, 0, 0, 0], dtype=np.int32)
    else:
        device = tensors[0].device
        assert len(tensors) <= 2
        a = tensors[0]
        b = tensors[1] if len(tensors) > 1 else None
        out = torch.empty(8, dtype=torch.int32, device=device)
        ws = workspace(lib().mn_map_workspace_bytes(0, 0, 0), device)
        _lib.check(lib().mn_bbox(ptr(a), a.shape[0], ptr(b), 0 if b is None else b.shape[0], ndim,
                                 ptr(out), ptr(ws), ws.numel(), stream_ptr(device)), "bbox")
        mm = out.cpu().numpy()
    _lib.check(lib().mn_keyspec_make(np_ptr(mm), ndim, max(int(num_clouds), 1), int(margin),
                                     ctypes.byref(spec)), "keyspec")
    return spec


def pack_keys(coords: torch.Tensor, batch_dims: Optional[torch.Tensor], spec: KeySpec,
              tstride: Optional[Sequence[int]] = None) -> torch.Tensor:
    n, ndim = coords.shape
    keys = torch.empty(n, dtype=torch.int64, device=coords.device)
    ts = None if tstride is None else np.asarray(tstride, dtype=np.int32)
    nb = 1 if batch_dims is None else batch_dims.numel() - 1
    _lib.check(lib().mn_pack_keys(ptr(coords), n, ndim, ptr(batch_dims), nb, np_ptr(ts),
                                  ctypes.byref(spec), ptr(keys), ptr(status_word(coords.device)),
                                  stream_ptr(coords.device)), "pack_keys")
    return keys


# ---------------------------------------------------------------------------
# plans of kernel maps (csrc/host.cpp:Plan): pair counts on the host, hit words,
# neighbour tables and pair lists, kept for as long as the mask tensors live
# ---------------------------------------------------------------------------
_plans = {}        # id(masks) or id(sizes) -> (weak reference, version, plan, side)
_foreign = {}      # (id(source masks), id(target masks)) of other maps -> (both references, versions, plan)
_host_copies = {}  # id(tensor) -> (weak reference, version, numpy values)
_SOURCE, _TARGET, _SIZES = range(3)


def version(*tensors):
    """Changes whenever one of ``tensors`` is written in place (None for tensors made in inference
    mode, which keep no count)."""
    try:
        return [t._version for t in tensors]
    except RuntimeError:
        return None


def _remember(t: torch.Tensor, plan, side: int):
    key = id(t)
    _plans[key] = (weakref.ref(t, lambda _r, k=key: _plans.pop(k, None)), version(t), plan, side)


def remember_plan(source_masks, target_masks, sizes, plan):
    """Find ``plan`` again by the tensors of its map, as long as nobody writes into them."""
    _remember(source_masks, plan, _SOURCE)
    _remember(target_masks, plan, _TARGET)
    _remember(sizes, plan, _SIZES)


def _entry(t: torch.Tensor):
    hit = _plans.get(id(t))
    return hit if hit is not None and hit[0]() is t and hit[1] == version(t) else None


def plan_of(source_masks: torch.Tensor, target_masks: torch.Tensor, sizes):
    """``(plan, swapped)`` of the map that two int32 mask tensors and its pair counts (a tensor or
    host values) describe; ``swapped`` when the masks are the map's own with the sides exchanged.
    Masks that did not come from this engine, or were written to since, get a plan of their own on
    first use; it serves until one of them is written to or other counts come with them."""
    s, t = _entry(source_masks), _entry(target_masks)
    own = s is not None and t is not None and s[2] is t[2] and s[3] != t[3]
    if own and isinstance(sizes, torch.Tensor):
        z = _entry(sizes)
        if z is not None and z[2] is s[2]:        # the map's own counts: no wait for their copy here
            return s[2], s[3] == _TARGET
    values = host_copy(sizes, np.int32) if isinstance(sizes, torch.Tensor) else np.asarray(sizes)
    values = values.tolist()
    if own and s[2].sizes() == values:
        return s[2], s[3] == _TARGET
    key = (id(source_masks), id(target_masks))
    versions = version(source_masks, target_masks)
    hit = _foreign.get(key)
    if hit is not None and hit[0]() is source_masks and hit[1]() is target_masks and \
            hit[2] == versions and hit[3].sizes() == values:
        return hit[3], False
    plan = _lib.host().Plan(source_masks.shape[0], source_masks.shape[1], target_masks.shape[1])
    plan.set_sizes(values)

    def drop(ref, k=key):
        if k in _foreign and any(r is ref for r in _foreign[k][:2]):
            del _foreign[k]

    _foreign[key] = (weakref.ref(source_masks, drop), weakref.ref(target_masks, drop), versions, plan)
    return plan, False


def remember_host(t: torch.Tensor, values: np.ndarray):
    key = id(t)
    _host_copies[key] = (weakref.ref(t, lambda _r, k=key: _host_copies.pop(k, None)), version(t), values)


def host_copy(t: torch.Tensor, dtype=np.int32) -> np.ndarray:
    """Host values of ``t``: the remembered copy when the tensor came from this
    engine, otherwise a blocking device-to-host read."""
    entry = _entry(t)
    if entry is not None and entry[3] == _SIZES:
        return np.asarray(entry[2].sizes(), dtype=dtype)
    hit = _host_copies.get(id(t))
    if hit is not None and hit[0]() is t and hit[1] == version(t):
        return np.ascontiguousarray(np.asarray(hit[2]).astype(dtype, copy=False))
    return np.ascontiguousarray(t.detach().cpu().numpy().astype(dtype, copy=False))


def hit_bits(masks: torch.Tensor) -> Optional[torch.Tensor]:
    """Hit words (bit p set <=> mask row p has an entry for the row) of a mask tensor that
    came from the fused map build, else None."""
    entry = _entry(masks)
    if entry is None or entry[3] == _SIZES:
        return None
    return entry[2].source_bits if entry[3] == _SOURCE else entry[2].target_bits


def neighbor_table(source_masks: torch.Tensor, target_masks: torch.Tensor,
                   sizes_host: np.ndarray, reorder: bool = True):
    """``(nbr [O, T] int32, tile_bits [ceil(T/128)] int32, perm [T] int32 or None)`` of
    the kernel map that the two mask tensors describe; built on first use and kept for
    as long as the masks live (a transposed convolution passes the same masks swapped
    and gets its own table).  With ``reorder`` and a map that carries hit words, the
    table's rows are the targets sorted by hit word (``perm[r]`` = target at position
    ``r``), so that 128-row tiles skip the offsets none of their rows has."""
    plan, swapped = plan_of(source_masks, target_masks, sizes_host)
    return plan.neighbours(swapped, reorder, source_masks, target_masks)
