"""Exact integer histogram of block-normalised gradients
(reference: kernels/exact_histogram_fused.py:10-58)."""
from __future__ import annotations

import numpy as np
import torch

from .. import _lib
from ._common import require_cuda_tensors, require_one_device


def gefen_exact_histogram_cuda(grad_flat: torch.Tensor, period: int, bin_counts: torch.Tensor) -> None:
    """bin_counts[b] += number of elements whose g/absmax(block) falls in bin b; int64, added to."""
    require_cuda_tensors({"grad_flat": grad_flat, "bin_counts": bin_counts})
    require_one_device("grad_flat and bin_counts", (grad_flat, bin_counts))
    if grad_flat.dim() != 1:
        raise ValueError("Expected grad_flat to be 1D, got dim={}".format(grad_flat.dim()))
    if bin_counts.dim() != 1:
        raise ValueError("Expected bin_counts to be 1D, got dim={}".format(bin_counts.dim()))
    if bin_counts.dtype != torch.int64:
        raise ValueError("Expected bin_counts to be int64, got {}".format(bin_counts.dtype))
    if period <= 0:
        raise ValueError("Expected period to be positive, got {}".format(period))
    if grad_flat.numel() % period != 0:
        raise ValueError("Expected grad_flat.numel()={} to be divisible by period={}.".format(
            grad_flat.numel(), period))
    if bin_counts.numel() <= 0 or bin_counts.numel() > 4096:
        raise ValueError("Expected histogram bins in [1, 4096], got {}".format(bin_counts.numel()))
    if not bin_counts.is_contiguous():
        raise ValueError("Expected bin_counts to be contiguous.")
    grad_flat = grad_flat.contiguous()
    with _lib.device_guard(grad_flat.device):
        _lib.check(_lib.load().gefen_b200_exact_histogram(
            _lib.ptr(grad_flat), _lib.dtype_tag(grad_flat.dtype), grad_flat.numel(), int(period),
            _lib.ptr(bin_counts), bin_counts.numel(), _lib.current_stream(grad_flat.device)))


def gefen_exact_histogram_many_cuda(grads_flat, periods, histogram_bins: int) -> torch.Tensor:
    """The float32 sum, in the given order, of the histograms of many contiguous 1-D gradients on one device, each
    converted to float32 first: one launch for all of them. Device tensor [histogram_bins]."""
    device = grads_flat[0].device
    require_one_device("the gradients of one histogram", grads_flat)
    require_cuda_tensors({"grad_flat {}".format(i): g for i, g in enumerate(grads_flat)})
    for g, period in zip(grads_flat, periods):
        if period <= 0 or g.numel() % period != 0:
            raise ValueError("Expected grad_flat.numel()={} to be divisible by period={}.".format(g.numel(), period))
    n = len(grads_flat)
    grads_flat = [g.contiguous() for g in grads_flat]
    lib = _lib.load()
    values = np.array([g.data_ptr() for g in grads_flat], dtype=np.uint64)
    dtypes = np.array([_lib.dtype_tag(g.dtype) for g in grads_flat], dtype=np.int32)
    numels = np.array([g.numel() for g in grads_flat], dtype=np.int64)
    lengths = np.array(periods, dtype=np.int64)
    rows = torch.empty((n, histogram_bins), dtype=torch.int64, device=device)
    total = torch.empty(histogram_bins, dtype=torch.float32, device=device)
    table = torch.empty(lib.gefen_b200_exact_histogram_many_table_bytes(n), dtype=torch.uint8, device=device)
    with _lib.device_guard(device):
        _lib.check(lib.gefen_b200_exact_histogram_many(
            n, values.ctypes.data, dtypes.ctypes.data, numels.ctypes.data, lengths.ctypes.data, _lib.ptr(rows),
            _lib.ptr(total), int(histogram_bins), _lib.ptr(table), _lib.current_stream(device)))
    return total
