"""Operands of multi-head latent attention: the query, key and value of softmax attention from the projections' outputs.

``mla_operands`` rotates the rotary part of every query head, appends the rotated rotary key (one for all heads) to every
head's own key part and separates the values, in one kernel forward and one backward (``csrc/mla.cu``). Tensors the
kernel does not take (CPU, other dtypes, widths that are no multiple of 8) go through the same steps in PyTorch, as do
forward-mode derivatives, the ``torch.func`` transforms, and gradients that are batched or differentiated again.
"""
from __future__ import annotations

import torch
from torch.autograd import forward_ad

from . import _lib
from ._lib import count_launch
from .elementwise import _rope_ref

_declared = False


def _ensure():
    global _declared
    if not _declared:
        import ctypes as c

        vp, i32, i64 = c.c_void_p, c.c_int, c.c_longlong
        _lib.declare("fsb_mla_pack", [vp] * 7 + [i64, i32, i32, i32, i32, i32, i64, vp])
        _lib.declare("fsb_mla_unpack", [vp] * 7 + [i64, i32, i32, i32, i32, i32, vp])
        _declared = True


def mla_operands_ref(q, kvb, k_pe, table, nope: int):
    """The same operands from PyTorch operations (differentiable)."""
    B, S, H, width = q.shape
    rope, value = width - nope, kvb.shape[-1] - nope
    k_nope, v = kvb.split([nope, value], dim=-1)
    q_nope, q_pe = q.split([nope, rope], dim=-1)
    q_pe = _rope_ref(q_pe, table, False)
    k_pe = _rope_ref(k_pe.reshape(B, S, 1, rope), table, False)
    return torch.cat([q_nope, q_pe], dim=-1), torch.cat([k_nope, k_pe.expand(B, S, H, rope)], dim=-1), v


def _grads_ref(dquery, dkey, dvalue, table, nope: int):
    """Gradients of the three inputs from PyTorch operations (a linear map, differentiable and batchable)."""
    dk_pe = _rope_ref(dkey[..., nope:].float().sum(2, keepdim=True), table, True).squeeze(2)
    return (torch.cat([dquery[..., :nope], _rope_ref(dquery[..., nope:], table, True)], dim=-1),
            torch.cat([dkey[..., :nope], dvalue], dim=-1), dk_pe.to(dkey.dtype))


class _MlaOperands(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, kvb, k_pe, table, nope):
        _ensure()
        B, S, H, width = q.shape
        rope, value = width - nope, kvb.shape[-1] - nope
        query, key = torch.empty_like(q), torch.empty_like(q)
        v = torch.empty(B, S, H, value, dtype=q.dtype, device=q.device)
        rc = _lib.load().fsb_mla_pack(q.data_ptr(), kvb.data_ptr(), k_pe.data_ptr(), table.data_ptr(), query.data_ptr(),
                                      key.data_ptr(), v.data_ptr(), B * S, S, H, nope, rope, value, k_pe.stride(1),
                                      _lib.stream_ptr(q.device))
        _lib.check(rc, "fsb_mla_pack")
        count_launch()
        ctx.save_for_backward(table)
        ctx.dims = (B, S, H, nope, rope, value)
        return query, key, v

    @staticmethod
    def backward(ctx, dquery, dkey, dvalue):
        (table,) = ctx.saved_tensors
        B, S, H, nope, rope, value = ctx.dims
        if torch.is_grad_enabled() or not _lib.plain(dquery, dkey, dvalue):
            return (*_grads_ref(dquery, dkey, dvalue, table, nope), None, None)
        dquery, dkey, dvalue = (g.contiguous() if g.data_ptr() % 16 == 0 else g.clone(memory_format=torch.contiguous_format)
                                for g in (dquery, dkey, dvalue))
        dq = torch.empty_like(dquery)
        dkvb = torch.empty(B, S, H, nope + value, dtype=dq.dtype, device=dq.device)
        dk_pe = torch.empty(B, S, rope, dtype=dq.dtype, device=dq.device)
        rc = _lib.load().fsb_mla_unpack(dquery.data_ptr(), dkey.data_ptr(), dvalue.data_ptr(), table.data_ptr(),
                                        dq.data_ptr(), dkvb.data_ptr(), dk_pe.data_ptr(), B * S, S, H, nope, rope, value,
                                        _lib.stream_ptr(dq.device))
        _lib.check(rc, "fsb_mla_unpack")
        count_launch()
        return dq, dkvb, dk_pe, None, None


def _native(q, kvb, k_pe, table, nope) -> bool:
    if not _lib.plain(q, kvb, k_pe, table) or forward_ad._current_level >= 0 or torch.compiler.is_compiling():
        return False
    B, S, H, width = q.shape
    rope, value = width - nope, kvb.shape[-1] - nope
    return (q.is_cuda and all(t.dtype == torch.bfloat16 and t.device == q.device for t in (q, kvb, k_pe))
            and table.dtype == torch.float32 and table.device == q.device and table.is_contiguous()
            and table.shape[0] >= S and table.shape[1] * 2 == rope
            and min(nope, rope, value) > 0 and nope % 8 == 0 and rope % 8 == 0 and value % 8 == 0
            and q.is_contiguous() and kvb.is_contiguous() and k_pe.dim() == 3 and k_pe.stride(2) == 1
            and k_pe.stride(0) == S * k_pe.stride(1) and k_pe.stride(1) % 8 == 0
            and all(t.data_ptr() % 16 == 0 for t in (q, kvb, k_pe, table)) and 0 < B * S < 2 ** 31)


def mla_operands(q, kvb, k_pe, table, nope: int):
    """``q`` [B, S, H, nope + rope], ``kvb`` [B, S, H, nope + value], ``k_pe`` [B, S, rope], ``table`` the rotary table
    [>= S, rope / 2, 2] -> query, key [B, S, H, nope + rope] and value [B, S, H, value]."""
    if _native(q, kvb, k_pe, table, nope):
        return _MlaOperands.apply(q, kvb, k_pe, table, nope)
    return mla_operands_ref(q, kvb, k_pe, table, nope)
