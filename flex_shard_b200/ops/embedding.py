"""Token embedding whose weight gradient is written once, into the reduction bucket where the weight has one.

The forward is PyTorch's gather. The backward (``csrc/embedding.cu``) adds the output gradients of equal tokens in fp32,
in an order that only the tokens decide, straight into the weight's ``main_grad`` view or a new gradient. Other weights
(CPU, other dtypes, widths) take PyTorch's backward.
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.autograd import forward_ad

from . import _lib
from ._lib import count_launch

_declared = False


def _ensure():
    global _declared
    if not _declared:
        import ctypes as c

        vp, i32, i64 = c.c_void_p, c.c_int, c.c_longlong
        _lib.declare("fsb_embedding_grad", [vp, vp, i32, i64, i32, i32, vp, i32, i32, vp, vp])
        _lib.declare("fsb_embedding_scratch_ints", [i64, i32, i32])
        _lib.load().fsb_embedding_scratch_ints.restype = i64
        _declared = True


def _write_grad(dy, tokens, out, accumulate: bool) -> None:
    _ensure()
    V, D = out.shape
    T = tokens.numel()
    lib = _lib.load()
    scratch = torch.empty(lib.fsb_embedding_scratch_ints(T, V, D), dtype=torch.int32, device=dy.device)
    rc = lib.fsb_embedding_grad(dy.data_ptr(), tokens.data_ptr(), int(tokens.dtype == torch.int64), T, V, D,
                                        out.data_ptr(), int(out.dtype == torch.float32), int(accumulate),
                                        scratch.data_ptr(), _lib.stream_ptr(dy.device))
    _lib.check(rc, "fsb_embedding_grad")
    count_launch(6 if T > 64 else 4)


def _hooked(weight) -> bool:
    return bool(weight._backward_hooks) or bool(getattr(weight, "_post_accumulate_grad_hooks", None))


class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, tokens, weight):
        ctx.save_for_backward(tokens)
        # a parameter's gradient destination is looked up when the gradient is there; a weight's values are not needed
        ctx.weight = weight if weight.is_leaf else None
        ctx.shape = weight.shape
        return F.embedding(tokens, weight)

    @staticmethod
    def backward(ctx, dy):
        (tokens,), weight = ctx.saved_tensors, ctx.weight
        if not ctx.needs_input_grad[1]:
            return None, None
        if torch.is_grad_enabled() or not _lib.plain(dy, tokens):
            # a gradient that is differentiated again, or batched gradients: the operator that autograd knows
            return None, torch.ops.aten.embedding_dense_backward(dy, tokens, ctx.shape[0], -1, False)
        tokens = tokens.reshape(-1).contiguous()
        dy = dy.reshape(-1, dy.shape[-1]).contiguous()
        if dy.data_ptr() % 16:
            dy = dy.clone()
        main = getattr(weight, "main_grad", None)
        if (isinstance(main, torch.Tensor) and main.dtype == torch.float32 and main.is_contiguous()
                and main.shape == ctx.shape and main.data_ptr() % 16 == 0 and not _hooked(weight)):
            _write_grad(dy, tokens, main, bool(getattr(weight, "main_grad_written", False)))
            weight.main_grad_written = True
            return None, None
        dw = torch.empty(ctx.shape, dtype=dy.dtype, device=dy.device)
        _write_grad(dy, tokens, dw, False)
        return None, dw


def embedding(tokens, weight):
    """Rows ``tokens`` (any shape, int32 or int64) of ``weight`` [V, D]. Forward-mode derivatives, the ``torch.func``
    transforms, tensor subclasses and compilers take PyTorch's operator."""
    if (_lib.plain(tokens, weight) and forward_ad._current_level < 0 and not torch.compiler.is_compiling()
            and weight.is_cuda and weight.dtype == torch.bfloat16 and weight.dim() == 2 and weight.shape[1] % 8 == 0
            and 0 < weight.shape[1] <= 8192 and weight.shape[0] > 0 and 0 < tokens.numel() < 2 ** 31
            and tokens.device == weight.device and tokens.dtype in (torch.int32, torch.int64)):
        return _Embedding.apply(tokens, weight)
    return F.embedding(tokens, weight)


class TokenEmbedding(nn.Embedding):
    """``nn.Embedding`` on ``embedding``; with a padding row, a norm limit, scaling by frequency or sparse gradients, PyTorch's.
    Where the gathered weight has a ``main_grad`` its gradient goes there and not through autograd (as with the products and
    norms of this library), unless the weight has hooks."""

    def forward(self, tokens):
        if self.padding_idx is not None or self.max_norm is not None or self.scale_grad_by_freq or self.sparse:
            return super().forward(tokens)
        return embedding(tokens, self.weight)
