"""Operations over many dense CUDA tensors at once (gradient norm, clipping): one launch per 96 tensors."""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._lib import count_launch

_declared = False


def _ensure():
    global _declared
    if not _declared:
        c = ctypes
        vp = c.c_void_p
        _lib.declare("fsb_sum_squares_scratch", [c.c_int])
        _lib.declare("fsb_sum_squares", [vp, vp, vp, c.c_int, vp, vp, vp])
        _lib.declare("fsb_clip_by_norm", [vp, vp, vp, c.c_int, vp, c.c_float, vp])
        _declared = True


def _lists(tensors):
    n = len(tensors)
    return ((ctypes.c_ulonglong * n)(*[t.data_ptr() for t in tensors]), (ctypes.c_longlong * n)(*[t.numel() for t in tensors]),
            (ctypes.c_int * n)(*[int(t.dtype == torch.float32) for t in tensors]), n)


def sum_squares(tensors) -> torch.Tensor:
    """fp32 sum of the squares of all elements of contiguous, non-empty bf16 / fp32 tensors of one GPU."""
    _ensure()
    lib = _lib.load()
    dev = tensors[0].device
    ptrs, sizes, fp32, n = _lists(tensors)
    scratch = torch.empty(lib.fsb_sum_squares_scratch(n), dtype=torch.float32, device=dev)
    out = torch.empty((), dtype=torch.float32, device=dev)
    with torch.cuda.device(dev):
        rc = lib.fsb_sum_squares(ptrs, sizes, fp32, n, scratch.data_ptr(), out.data_ptr(), _lib.stream_ptr(dev))
    _lib.check(rc, "fsb_sum_squares")
    count_launch(1 + -(-n // 96))
    return out


def clip_by_norm_(tensors, norm: torch.Tensor, max_norm: float) -> None:
    """Scales the tensors in place by ``min(1, max_norm / (norm + 1e-6))``; ``norm`` is an fp32 scalar on their GPU."""
    _ensure()
    dev = tensors[0].device
    ptrs, sizes, fp32, n = _lists(tensors)
    with torch.cuda.device(dev):
        rc = _lib.load().fsb_clip_by_norm(ptrs, sizes, fp32, n, norm.data_ptr(), float(max_norm), _lib.stream_ptr(dev))
    _lib.check(rc, "fsb_clip_by_norm")
    torch.autograd.graph.increment_version(tensors)
    count_launch(-(-n // 96))
