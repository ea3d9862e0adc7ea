"""Voxelisation: float points -> sorted unique integer voxels
(the step before the hot path; API of minuet/nn/functional/voxelize.py)."""
__all__ = ['voxelize']

from typing import Optional

import numpy as np
import torch

from minuet_b200 import _lib, engine
from minuet_b200.nn.functional.hash import unique_coordinates
from minuet_b200.nn.functional.indexing import build_sorted_index


def voxelize(coordinates: torch.Tensor, voxel_size, batch_dims: Optional[torch.Tensor] = None,
             return_inverse: bool = False, features: Optional[torch.Tensor] = None):
    """Floor ``coordinates / voxel_size`` to int32 voxels, sort them (cloud-major,
    then lexicographically) and drop duplicates.

    Returns ``(voxels [U, D], batch_dims [B + 1] or None)`` and, with
    ``return_inverse``, also ``inverse [N]`` such that ``voxels[inverse[i]]`` is the
    voxel of input point ``i``.  With ``features [N, C]`` (fp32 / fp16 / bf16) the
    result also carries ``voxel_features [U, C]``, the mean of the features of the
    points of every voxel (one kernel over the sorted runs, fp32 sums in a fixed
    order), appended last: ``(voxels, batch_dims[, inverse], voxel_features)``.

    The reference's function has the same purpose but cannot run as shipped (it
    passes a dtype as ``device=`` and skips the sort that its unique step needs,
    minuet/nn/functional/voxelize.py:10-35); this one follows the documented
    intent: floor, sort, unique.
    """
    if coordinates.ndim != 2:
        raise ValueError(f"coordinates must be [N, D] but found {coordinates.ndim}-D")
    engine.require_cuda(coordinates, batch_dims)
    if features is not None and (features.ndim != 2 or features.shape[0] != coordinates.shape[0]):
        raise ValueError("features must be [N, C] with one row per point")
    engine.require_cuda(features)
    native = _native(coordinates, voxel_size, batch_dims, return_inverse, features)
    if native is not None:
        return native
    # other point types, sizes in tensors, boxes too wide for one key: step by step
    size = torch.as_tensor(voxel_size, dtype=coordinates.dtype, device=coordinates.device)
    voxels = torch.floor(coordinates / size).to(torch.int32)
    index = build_sorted_index(voxels, batch_dims=batch_dims)
    sorted_voxels = voxels[index]
    unique, indices = unique_coordinates(sorted_voxels, batch_dims=batch_dims)
    new_batch_dims = None
    if batch_dims is not None:
        new_batch_dims = indices[batch_dims.to(torch.int64)].to(batch_dims.dtype)
    result = [unique, new_batch_dims]
    run_ids = indices[:-1].to(torch.int64).contiguous()
    if return_inverse:
        # indices[i] = runs closed before sorted row i = the unique voxel of that row; undo the sort
        inverse = torch.empty(voxels.shape[0], dtype=torch.int64, device=voxels.device)
        inverse[index] = run_ids
        result.append(inverse)
    if features is not None:
        feats = features.contiguous()
        means = torch.empty((unique.shape[0], feats.shape[1]), dtype=feats.dtype,
                            device=feats.device)
        _lib.check(engine.lib().mn_voxel_mean(
            engine.ptr(feats), feats.shape[0], feats.shape[1], engine.dtype_code(feats.dtype),
            engine.ptr(index.to(torch.int64).contiguous()), engine.ptr(run_ids), engine.ptr(means),
            engine.stream_ptr(feats.device)), "voxel_mean")
        result.append(means)
    return tuple(result)


def _native(coordinates, voxel_size, batch_dims, return_inverse, features):
    """The whole of it in a handful of launches and one read of the number of voxels; None
    where that path does not apply."""
    n, ndim = coordinates.shape
    if not coordinates.is_cuda or coordinates.dtype not in (torch.float32, torch.float64) or \
            n == 0 or ndim > _lib.MN_MAX_NDIM or isinstance(voxel_size, torch.Tensor):
        return None
    if features is not None and (features.shape[1] == 0 or features.dtype not in (
            torch.float32, torch.float16, torch.bfloat16)):
        return None
    # one size or one per dimension; whatever else broadcasts, or is refused, goes step by step
    if type(voxel_size) is float:
        sizes = [voxel_size] * ndim
    else:
        try:
            if np.ndim(voxel_size) > 1:
                return None
            sizes = [float(v) for v in (voxel_size if hasattr(voxel_size, "__len__") else (voxel_size,))]
        except (TypeError, ValueError):
            return None
        if len(sizes) == 1:
            sizes = sizes * ndim
        if len(sizes) != ndim:
            return None
    out = _lib.host().voxelize(coordinates.detach(), sizes, engine.as_i64(batch_dims), return_inverse,
                               features)
    if out is None:
        return None
    voxels, starts, inverse, means = out
    result = [voxels, None if batch_dims is None else starts.to(batch_dims.dtype)]
    if return_inverse:
        result.append(inverse)
    if features is not None:
        result.append(means)
    return tuple(result)
