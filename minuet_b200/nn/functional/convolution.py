"""Gather - grouped GEMM - Scatter forward pass and its stage timers
(mirror of minuet/nn/functional/convolution.py)."""
__all__ = ['cuda_time_gather', 'cuda_time_scatter', 'sparse_convolution_forward',
           'sparse_convolution_forward_fused', 'apply_epilogue', 'cuda_time_gemm',
           'set_gemm_parallel_level', 'dense_forward', 'time_forward', 'estimate_ms',
           'transpose_weights']

from typing import Optional

import numpy as np
import torch

from minuet_b200 import _lib, engine

GEMM_PARALLEL_LEVEL = 4
# Which forward algorithm fp16/bf16 layers use when the call does not say:
# "explicit" = pair lists (or gather - grouped GEMM - scatter where pair lists do not
# apply), "implicit" = the fused output-stationary kernel, "auto" = a cost estimate
# from the map's pair and tile counts (no timing ever runs inside a forward pass; the
# layer autotuner times both and passes its choice with every call)
ALGORITHM = "auto"
# 128-row sub-tiles per CTA tile of the fused kernel when the call does not say
# (0 = chosen by the library)
IMPLICIT_SUB_TILES = 0
# The fused kernel walks the targets sorted by hit word (rows with the same set of
# offsets share tiles, and tiles skip the offsets they do not have); False keeps the
# targets' own order
REORDER_ROWS = True


def set_gemm_parallel_level(level: int):
    """Kept for API compatibility (minuet/nn/functional/convolution.py:15-25).
    The reference spreads one cuBLAS call per padding bucket over ``level``
    streams; here every offset is a problem of one grouped launch, so the value
    is stored and otherwise unused."""
    global GEMM_PARALLEL_LEVEL
    GEMM_PARALLEL_LEVEL = level


def _i32(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    if t is None:
        return None
    return t.contiguous() if t.dtype == torch.int32 else t.to(torch.int32).contiguous()


def _prepare(weights, source_masks, target_masks, kernel_map_sizes, sources=None):
    if source_masks.ndim != 2 or target_masks.ndim != 2:
        raise RuntimeError("source_masks and target_masks must be 2-D tensors")
    if weights.ndim != 3:
        raise RuntimeError(f"weights must be a 3-D tensor but found {weights.ndim}-D")
    O, T = target_masks.shape
    S = source_masks.shape[1]
    if source_masks.shape[0] != O or weights.shape[0] != O or kernel_map_sizes.shape[0] != O:
        raise RuntimeError("source_masks, weights and kernel_map_sizes must have one row per "
                           f"offset ({O})")
    c_in, c_out = weights.shape[1], weights.shape[2]
    if sources is not None:
        if sources.ndim != 2 or sources.shape[1] != c_in:
            raise RuntimeError(f"sources must be [N, {c_in}] but found {tuple(sources.shape)}")
        if sources.dtype != weights.dtype:
            raise RuntimeError(f"sources ({sources.dtype}) and weights ({weights.dtype}) must "
                               "share one dtype")
    sizes_host = engine.host_copy(kernel_map_sizes, np.int32)
    return S, T, O, c_in, c_out, sizes_host


_ALGORITHMS = {"auto": 0, "explicit": 1, "implicit": 2}


def native_options(gather_tile_size, scatter_tile_size, allow_shortcut_matmul, threshold, algorithm,
                   sub_tiles, relu):
    """The options of a call in native form; the module-level choices stand in where the call
    makes none."""
    if algorithm in (None, "auto"):
        algorithm = ALGORITHM
    if algorithm not in _ALGORITHMS:
        raise ValueError(f"unknown sparse convolution algorithm {algorithm!r}")
    return _lib.host().ConvOptions(
        bool(allow_shortcut_matmul), _ALGORITHMS[algorithm],
        int(IMPLICIT_SUB_TILES if sub_tiles is None else sub_tiles), int(gather_tile_size),
        int(scatter_tile_size), None if threshold is None else float(threshold), REORDER_ROWS,
        bool(relu))


def run(plan, swapped, sources, weights, source_masks, target_masks, order, options, weights_t=None):
    """A planned forward pass (see ``engine.plan_of``), differentiable where it has to be."""
    if torch.is_grad_enabled() and (sources.requires_grad or weights.requires_grad):
        return _lib.host().conv_autograd(plan, swapped, sources, weights, source_masks, target_masks,
                                         order, options)
    return run_fused(plan, swapped, sources, weights, source_masks, target_masks, order, options,
                     weights_t)


def run_fused(plan, swapped, sources, weights, source_masks, target_masks, order, options,
              weights_t=None, scale=None, shift=None, residual=None):
    """A planned forward pass with the epilogue inside, not differentiable."""
    log = engine.LAYER_LOG
    if log is None:
        return _lib.host().conv_forward(plan, swapped, sources, weights, source_masks, target_masks,
                                        order, weights_t, scale, shift, residual, options)
    c_in, c_out = weights.shape[1], weights.shape[2]
    if weights.dtype != torch.float32 and c_in % 8 and c_out % 8 == 0:
        c_in += -c_in % 8          # runs zero-padded
    entry = {"S": source_masks.shape[1], "T": target_masks.shape[1], "O": source_masks.shape[0],
             "E": plan.pairs(), "c_in": c_in, "c_out": c_out,
             "events": engine.event_pair_begin(sources.device)}
    log.append(entry)
    out = _lib.host().conv_forward(plan, swapped, sources, weights, source_masks, target_masks, order,
                                   weights_t, scale, shift, residual, options)
    engine.event_pair_end(entry["events"], sources.device)
    entry["algorithm"] = "implicit" if plan.last_algorithm == 2 else "explicit"
    if entry["algorithm"] == "implicit":      # the per-tile offset bits of the logged layer
        entry["tile_bits"] = plan.neighbours(swapped, REORDER_ROWS, source_masks, target_masks)[1]
    return out


def _workspace(sizes_host, S, T, O, c_in, c_out, code, allow_shortcut, threshold, device):
    nbytes = engine.lib().mn_conv_workspace_bytes(
        engine.np_ptr(sizes_host), O, S, T, c_in, c_out, code, int(bool(allow_shortcut)),
        0 if threshold is None else 1, 0.0 if threshold is None else float(threshold))
    return engine.workspace(nbytes, device)


def sparse_convolution_forward(sources: torch.Tensor,
                               weights: torch.Tensor,
                               source_masks: torch.Tensor,
                               target_masks: torch.Tensor,
                               kernel_map_order: Optional[torch.Tensor],
                               kernel_map_sizes: torch.Tensor,
                               gather_tile_size: int,
                               scatter_tile_size: int,
                               allow_shortcut_matmul: bool = False,
                               parallel: Optional[int] = None,
                               threshold: Optional[float] = 0,
                               algorithm: Optional[str] = None,
                               sub_tiles: Optional[int] = None,
                               weights_t: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[t] = sum_k sum_{(s, t) in map[k]} sources[s] @ weights[order[k]]``
    (minuet/nn/functional/convolution.py:110-155).

    Arguments and result follow the reference; fp32, fp16 and bf16 features are
    supported (accumulation is always fp32).  ``parallel`` and ``threshold`` are
    accepted and do not change the result: the grouped GEMM needs neither side
    streams nor equal-size buckets.  ``*_tile_size`` is the number of channels
    one thread moves per row; 1 (the untuned default) picks 16-byte accesses.
    fp16/bf16 layers run either the pair-list forward or the fused implicit-GEMM
    kernel: ``algorithm`` ("explicit" / "implicit"; default: the module-level
    ``ALGORITHM``) and ``sub_tiles`` (row sub-tiles per tile of the fused kernel,
    0 = automatic) are this library's additions to the reference signature and are
    what the layer autotuner tunes; ``weights_t`` is :func:`transpose_weights` of
    ``weights`` for callers whose weights do not change between calls (without it the
    16-bit paths transpose the weights on every call).  Differentiable in ``sources`` and
    ``weights`` (the reference has no backward pass).
    """
    del parallel
    engine.require_cuda(sources)
    sm, tm, order = _i32(source_masks), _i32(target_masks), _i32(kernel_map_order)
    sizes_host = _prepare(weights, sm, tm, kernel_map_sizes)[-1]
    plan, swapped = engine.plan_of(sm, tm, sizes_host)
    options = native_options(gather_tile_size, scatter_tile_size, allow_shortcut_matmul, threshold,
                             algorithm, sub_tiles, False)
    return run(plan, swapped, sources, weights, sm, tm, order, options, weights_t)


def sparse_convolution_forward_fused(sources: torch.Tensor, weights: torch.Tensor,
                                     source_masks: torch.Tensor, target_masks: torch.Tensor,
                                     kernel_map_order: Optional[torch.Tensor],
                                     kernel_map_sizes: torch.Tensor,
                                     gather_tile_size: int = 1,
                                     scatter_tile_size: int = 1,
                                     allow_shortcut_matmul: bool = False,
                                     threshold: Optional[float] = 0,
                                     scale: Optional[torch.Tensor] = None,
                                     shift: Optional[torch.Tensor] = None,
                                     residual: Optional[torch.Tensor] = None,
                                     relu: bool = False,
                                     algorithm: Optional[str] = None,
                                     sub_tiles: Optional[int] = None,
                                     weights_t: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Sparse convolution with a fused epilogue (no counterpart in the reference,
    whose models apply BatchNorm, the residual add and ReLU as separate passes
    over the feature matrix):

        out = relu?( conv(sources) * scale[c] + shift[c] + residual )

    ``scale`` / ``shift`` are ``[C_out]`` (an eval-mode BatchNorm or a bias folded
    into two vectors; applied in fp32), ``residual`` is ``[N_out, C_out]`` in the
    feature dtype.  Layers that take the fused implicit-GEMM kernel apply the
    epilogue inside it; the others run gather - GEMM - scatter and one in-place
    pass over the output."""
    engine.require_cuda(sources)
    sm, tm, order = _i32(source_masks), _i32(target_masks), _i32(kernel_map_order)
    sizes_host = _prepare(weights, sm, tm, kernel_map_sizes)[-1]
    plan, swapped = engine.plan_of(sm, tm, sizes_host)
    options = native_options(gather_tile_size, scatter_tile_size, allow_shortcut_matmul, threshold,
                             algorithm, sub_tiles, relu)
    return run_fused(plan, swapped, sources, weights, sm, tm, order, options, weights_t, scale,
                     shift, residual)


def apply_epilogue(features: torch.Tensor, scale=None, shift=None, residual=None,
                   relu: bool = False) -> torch.Tensor:
    """In place ``features = relu?(features * scale[c] + shift[c] + residual)``."""
    engine.require_cuda(features, scale, shift, residual)
    rows, channels = features.shape
    _lib.check(engine.lib().mn_apply_epilogue(
        engine.ptr(features), rows, channels, engine.dtype_code(features.dtype),
        engine.ptr(_f32(scale)), engine.ptr(_f32(shift)),
        engine.ptr(None if residual is None else residual.contiguous()), int(bool(relu)),
        engine.stream_ptr(features.device)), "apply_epilogue")
    return features


def _f32(v):
    return None if v is None else v.detach().to(torch.float32).contiguous()


def transpose_weights(weights: torch.Tensor) -> Optional[torch.Tensor]:
    """``weights [O, c_in, c_out]`` (or ``[c_in, c_out]``) as ``[O, c_out, c_in]``, the
    layout the tensor-core kernels read; None for dtypes those kernels do not take."""
    if weights.dtype not in (torch.float16, torch.bfloat16) or not weights.is_cuda:
        return None
    w = weights.detach().contiguous()
    if w.ndim == 2:
        w = w.unsqueeze(0)
    O, c_in, c_out = w.shape
    out = torch.empty((O, c_out, c_in), dtype=w.dtype, device=w.device)
    _lib.check(engine.lib().mn_transpose_weights(
        engine.ptr(w), O, c_in, c_out, engine.dtype_code(w.dtype), engine.ptr(out),
        engine.stream_ptr(w.device)), "transpose_weights")
    return out


def dense_forward(features, weight, scale=None, shift=None, residual=None, relu=False,
                  weights_t=None):
    """``relu?((features @ weight) * scale + shift + residual)`` for a 1x1x1
    convolution: the tensor-core GEMM of this library for fp16/bf16 (c_in a multiple
    of 8, c_out even, at most 256), its FFMA GEMM plus the epilogue pass otherwise
    (fp32 must not go through TF32: its 10-bit mantissa would break the 1e-5 bound)."""
    engine.require_cuda(features)
    if features.dtype != weight.dtype or features.dtype not in (torch.float32, torch.float16,
                                                                 torch.bfloat16):
        raise RuntimeError(f"features ({features.dtype}) and weight ({weight.dtype}) must share "
                           "one of float32, float16, bfloat16")
    log = engine.LAYER_LOG
    if log is None:
        return _lib.host().dense_forward(features, weight, scale, shift, residual, bool(relu),
                                         weights_t)[0]
    entry = {"S": features.shape[0], "T": features.shape[0], "O": 1, "E": features.shape[0],
             "c_in": features.shape[1], "c_out": weight.shape[1],
             "events": engine.event_pair_begin(features.device)}
    log.append(entry)
    out, tensor_core = _lib.host().dense_forward(features, weight, scale, shift, residual,
                                                 bool(relu), weights_t)
    engine.event_pair_end(entry["events"], features.device)
    entry["algorithm"] = "dense" if tensor_core else "dense-ffma"
    return out


def estimate_ms(algorithm: str, S, T, O, c_in, c_out, pairs, shortcut: bool) -> float:
    """Rough cost of one 16-bit forward pass with an algorithm, in milliseconds (the estimate
    behind the automatic choice; only the order of two estimates matters)."""
    return _lib.host().estimate_ms(algorithm == "implicit", S, T, O, c_in, c_out, pairs,
                                   bool(shortcut), REORDER_ROWS)


def time_forward(weights, source_masks, target_masks, kernel_map_order, kernel_map_sizes,
                 allow_shortcut_matmul: bool = False, algorithm: str = "explicit",
                 sub_tiles: int = 0, gather_tile_size: int = 1, scatter_tile_size: int = 1,
                 threshold: Optional[float] = -1, epilogue=(False, False, False, False)) -> float:
    """Milliseconds of one whole forward pass with the given algorithm on buffers whose
    contents do not matter (what the layer autotuner compares).  ``epilogue`` =
    (scale, shift, residual, relu) flags of the fused epilogue the layer runs with."""
    engine.require_cuda(weights, source_masks, target_masks)
    weights = weights.detach().contiguous()
    sm, tm, order = _i32(source_masks), _i32(target_masks), _i32(kernel_map_order)
    S, T, O, c_in, c_out, sizes_host = _prepare(weights, sm, tm, kernel_map_sizes)
    device = weights.device
    sources = torch.zeros((S, c_in), dtype=weights.dtype, device=device)
    scale = torch.ones(c_out, dtype=torch.float32, device=device) if epilogue[0] else None
    shift = torch.zeros(c_out, dtype=torch.float32, device=device) if epilogue[1] else None
    residual = torch.zeros((T, c_out), dtype=weights.dtype, device=device) if epilogue[2] else None
    stream = torch.cuda.current_stream(device)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    plan, swapped = engine.plan_of(sm, tm, sizes_host)
    options = native_options(gather_tile_size, scatter_tile_size, allow_shortcut_matmul, threshold,
                             algorithm, sub_tiles, bool(epilogue[3]))
    begin.record(stream)
    run_fused(plan, swapped, sources, weights, sm, tm, order, options, None, scale, shift, residual)
    end.record(stream)
    end.synchronize()
    return begin.elapsed_time(end)


def _time_stage(stage, weights, source_masks, target_masks, kernel_map_sizes, tile_size,
                allow_shortcut_matmul, threshold) -> float:
    engine.require_cuda(weights, source_masks, target_masks)
    weights = weights.detach().contiguous()
    sm, tm = _i32(source_masks), _i32(target_masks)
    S, T, O, c_in, c_out, sizes_host = _prepare(weights, sm, tm, kernel_map_sizes)
    code = engine.dtype_code(weights.dtype)
    device = weights.device
    # like the reference's timers (sparse_convolution.cu:294-502) the stage runs
    # on buffers whose contents do not matter
    sources = torch.empty((S, c_in), dtype=weights.dtype, device=device)
    out = torch.empty((T, c_out), dtype=weights.dtype, device=device)
    ws = _workspace(sizes_host, S, T, O, c_in, c_out, code, allow_shortcut_matmul, threshold, device)
    stream = torch.cuda.current_stream(device)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record(stream)
    _lib.check(engine.lib().mn_conv_stage(
        stage, S, T, O, c_in, c_out, code, engine.ptr(sources), engine.ptr(weights),
        engine.ptr(sm), engine.ptr(tm), None, engine.np_ptr(sizes_host), int(tile_size),
        int(bool(allow_shortcut_matmul)), 0 if threshold is None else 1,
        0.0 if threshold is None else float(threshold), engine.ptr(out),
        engine.ptr(engine.status_word(device)), engine.ptr(ws), ws.numel(),
        engine.stream_ptr(device)), "conv_stage")
    end.record(stream)
    end.synchronize()
    return begin.elapsed_time(end)


def cuda_time_gather(weights, source_masks, target_masks, kernel_map_sizes, tile_size: int,
                     allow_shortcut_matmul: bool = False, threshold: float = 0) -> float:
    """Milliseconds of one gather (minuet/nn/functional/convolution.py:28-52)."""
    return _time_stage(0, weights, source_masks, target_masks, kernel_map_sizes, tile_size,
                       allow_shortcut_matmul, threshold)


def cuda_time_scatter(weights, source_masks, target_masks, kernel_map_sizes, tile_size: int,
                      allow_shortcut_matmul: bool = False, threshold: float = 0) -> float:
    """Milliseconds of one scatter (minuet/nn/functional/convolution.py:55-79)."""
    return _time_stage(2, weights, source_masks, target_masks, kernel_map_sizes, tile_size,
                       allow_shortcut_matmul, threshold)


def cuda_time_gemm(weights, source_masks, target_masks, kernel_map_sizes,
                   allow_shortcut_matmul: bool = False, parallel: Optional[int] = None,
                   threshold: float = 0) -> float:
    """Milliseconds of the grouped GEMM (minuet/nn/functional/convolution.py:82-107)."""
    del parallel
    return _time_stage(1, weights, source_masks, target_masks, kernel_map_sizes, 1,
                       allow_shortcut_matmul, threshold)
