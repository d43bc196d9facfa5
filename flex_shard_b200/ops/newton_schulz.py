"""Newton-Schulz orthogonalisation on the tcgen05 GEMM, with the polynomial fused in epilogues.

Per step (coefficients a, b, c), for ``X`` of shape ``[s, l]`` with ``s <= l``::

    A = X X^T                      one GEMM
    B = b*A + c*A@A                one GEMM, epilogue  c*acc + b*A
    X = a*X + B@X                  one GEMM, epilogue  acc + a*X

Tall matrices use ``A = X^T X`` and ``X = a*X + X@B`` instead, through the GEMM's transposed
operand modes, so no transpose copy is ever made. ``A`` and ``B`` are symmetric: their GEMMs compute the
tiles on or above the diagonal only and mirror them (28 % fewer FLOPs per iteration for a 4096 x 14336 matrix). Math parity with the reference's
``_zeropower_via_newtonschulz`` (``dist_muon/optimizer.py:2120-2151``): bf16 operands, fp32
accumulation, Frobenius normalisation first.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._lib import count_launch
from .gemm import gemm

NS_COEFFS = (3.4445, -4.7750, 2.0315)
_declared = False


def _ensure():
    global _declared
    if not _declared:
        c = ctypes
        vp, i32, i64, f32 = c.c_void_p, c.c_int, c.c_longlong, c.c_float
        _lib.declare("fsb_muon_prepare", [vp, vp, i32, vp, vp, i64, i32, f32, i32, vp])
        _lib.declare("fsb_muon_sum_squares", [vp, vp, i64, i32, vp])
        _lib.declare("fsb_muon_scale", [vp, vp, i32, i64, i32, f32, i32, vp])
        _lib.declare("fsb_muon_update", [vp, i32, vp, i64, f32, f32, vp])
        _lib.declare("fsb_muon_workspace_floats", [i64, i32])
        _lib.declare("fsb_gemm_pairs_usable", [])
        _lib.declare("fsb_gemm_bf16_batched", [vp, vp, vp, vp, i32, i32, i32, i32, i32, i32, f32, f32, i32, vp, vp])
        _declared = True


def _workspace(device, n: int, count: int = 1) -> torch.Tensor:
    """Zeroed scratch ``[count, floats]`` of the prepare kernel for ``count`` matrices of ``n`` elements: [m, 0] receives
    matrix m's sum of squares, the rest of its row holds the per-block partial sums, which the matrix's last block adds
    in index order (the same bits on every run)."""
    floats = _lib.load().fsb_muon_workspace_floats(n, count)
    return torch.zeros(count, floats // count, dtype=torch.float32, device=device)


def ns_iterations(x: torch.Tensor, steps: int = 5, coeffs=NS_COEFFS) -> torch.Tensor:
    """Run the iteration on an already normalised bf16 matrix ``x`` (any aspect ratio)."""
    a, b, c = coeffs
    rows, cols = x.shape
    wide = rows <= cols
    s = min(rows, cols)
    A = torch.empty(s, s, dtype=x.dtype, device=x.device)
    B = torch.empty(s, s, dtype=x.dtype, device=x.device)
    nxt = torch.empty_like(x)
    for _ in range(steps):
        if wide:
            gemm(x, x, out=A, symmetric=True)                   # A = X X^T
            gemm(A, A, out=B, c=A, alpha=c, beta=b, symmetric=True)   # B = b A + c A A   (A symmetric)
            gemm(B, x, b_t=True, out=nxt, c=x, alpha=1.0, beta=a)  # X = a X + B X
        else:
            gemm(x, x, a_t=True, b_t=True, out=A, symmetric=True)     # A = X^T X
            gemm(A, A, out=B, c=A, alpha=c, beta=b, symmetric=True)
            gemm(x, B, out=nxt, c=x, alpha=1.0, beta=a)         # X = a X + X B     (B symmetric)
        x, nxt = nxt, x
    return x


def _batched(a, b, out, M, N, K, *, a_t=False, b_t=False, c=None, alpha=1.0, beta=0.0, symmetric=False):
    """One product for every matrix of contiguous stacks: ``out[e] = alpha * A[e] @ B[e]^T + beta * c[e]``."""
    _ensure()
    rc = _lib.load().fsb_gemm_bf16_batched(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), c.data_ptr() if c is not None else None, a.shape[0], M, N, K,
        int(a_t), int(b_t), alpha, beta, int(symmetric), _lib.status_word(a.device).data_ptr(), _lib.stream_ptr(a.device))
    _lib.check(rc, "fsb_gemm_bf16_batched")
    count_launch()


def batched_ns_supported(x: torch.Tensor) -> bool:
    """Stacks of equal matrices whose dimensions are multiples of 8 (16-byte rows, which the copy engine needs) run every
    product of an iteration as one launch over the whole stack, where SM pairs can be used. Others take a matrix at a
    time."""
    if not (x.is_cuda and x.dim() == 3 and 1 < x.shape[0] <= 65535 and x.shape[1] % 8 == 0 and x.shape[2] % 8 == 0
            and x.numel() > 0):
        return False
    _ensure()
    return bool(_lib.load().fsb_gemm_pairs_usable())


def ns_iterations_batched(x: torch.Tensor, steps: int = 5, coeffs=NS_COEFFS) -> torch.Tensor:
    """The iteration on a stack ``[E, rows, cols]`` of normalised bf16 matrices: three GEMM launches per step for all
    ``E`` matrices (per-head and per-expert matrices are small; one launch each would leave most of the GPU idle and pay
    15 launches per matrix).  Same arithmetic per matrix as ``ns_iterations``."""
    a, b, c = coeffs
    E, rows, cols = x.shape
    wide = rows <= cols
    s = min(rows, cols)
    x = x.contiguous()
    A = torch.empty(E, s, s, dtype=x.dtype, device=x.device)
    B = torch.empty_like(A)
    nxt = torch.empty_like(x)
    for _ in range(steps):
        if wide:
            _batched(x, x, A, s, s, cols, symmetric=True)                                # A = X X^T
            _batched(A, A, B, s, s, s, c=A, alpha=c, beta=b, symmetric=True)             # B = b A + c A A
            _batched(B, x, nxt, s, cols, s, b_t=True, c=x, beta=a)                       # X = a X + B X
        else:
            _batched(x, x, A, s, s, rows, a_t=True, b_t=True, symmetric=True)            # A = X^T X
            _batched(A, A, B, s, s, s, c=A, alpha=c, beta=b, symmetric=True)
            _batched(x, B, nxt, rows, s, s, c=x, beta=a)                                 # X = a X + X B
        x, nxt = nxt, x
    return x


def _newton_schulz_cpu(g: torch.Tensor, steps: int, coeffs, eps: float) -> torch.Tensor:
    """The CPU statement of the iteration, in the very operations ``torch.optim.Muon`` uses (bf16 norm and division,
    bf16 ``matmul`` / ``addmm``), so that on CPU an owner-stored matrix steps bitwise like that optimizer."""
    a, b, c = coeffs
    x = g.to(torch.bfloat16)
    tall = g.size(0) > g.size(1)
    if tall:
        x = x.T
    x = x / x.norm().clamp(min=eps)
    for _ in range(steps):
        gram = x @ x.T
        x = torch.addmm(x, torch.addmm(gram, gram, gram, beta=b, alpha=c), x, beta=a)
    return x.T if tall else x


def newton_schulz_kernel_reference(g: torch.Tensor, steps: int = 5, coeffs=NS_COEFFS, eps: float = 1e-7) -> torch.Tensor:
    """CPU restatement of the arithmetic of the GPU kernels for one matrix (norm in fp32, the scaled matrix rounded to
    bf16 once, every product accumulated in fp32 and rounded once): the oracle the GPU tests compare against."""
    x = g.detach().cpu().to(torch.bfloat16)
    x = x / x.float().norm().clamp_min(eps).to(torch.bfloat16)
    return ns_iterations(x.contiguous(), steps, coeffs)


def newton_schulz(g: torch.Tensor, steps: int = 5, coeffs=NS_COEFFS, eps: float = 1e-7) -> torch.Tensor:
    """Approximate polar factor of ``g`` ([rows, cols] or batched [n, rows, cols]); returns bf16."""
    if g.dim() == 2 and not g.is_cuda:
        return _newton_schulz_cpu(g, steps, coeffs, eps)
    if g.dim() == 3:
        if batched_ns_supported(g):
            x = g.to(torch.bfloat16)
            norm = x.float().square().sum((1, 2), keepdim=True).sqrt().clamp_min(eps)
            return ns_iterations_batched((x.float() / norm).to(torch.bfloat16), steps, coeffs)
        return torch.stack([newton_schulz(m, steps, coeffs, eps) for m in g])
    x = g.to(torch.bfloat16)
    x = x / x.float().norm().clamp_min(eps).to(torch.bfloat16) if not x.is_cuda else _normalise_cuda(x, eps)
    return ns_iterations(x.contiguous(), steps, coeffs)


def _normalise_cuda(x: torch.Tensor, eps: float) -> torch.Tensor:
    _ensure()
    x = x.contiguous().clone()
    ss = (x.float() ** 2).sum().reshape(1)
    return _normalise_(x, ss.view(1, 1), eps)


def _normalise_(u: torch.Tensor, ws: torch.Tensor, eps: float) -> torch.Tensor:
    """Divides every matrix of ``u`` by its norm in place, whose square is in ``ws[m, 0]`` (a workspace as ``_workspace``
    gives it). Stacks divide element by element; a single matrix is multiplied by the norm's reciprocal."""
    _ensure()
    count = u.shape[0] if u.dim() == 3 else 1
    rc = _lib.load().fsb_muon_scale(u.data_ptr(), ws.data_ptr(), ws.shape[1], u.numel() // count, count, eps,
                                    int(u.dim() == 3), _lib.stream_ptr(u.device))
    _lib.check(rc, "fsb_muon_scale")
    count_launch()
    return u


def _sum_squares(u: torch.Tensor) -> torch.Tensor:
    """Workspace with the squared norms of the matrices of a contiguous bf16 stack: the bits that ``_prepare`` leaves
    when it makes the stack (of matrices on 16-byte boundaries), however many matrices the stack has."""
    _ensure()
    ws = _workspace(u.device, u[0].numel(), u.shape[0])
    rc = _lib.load().fsb_muon_sum_squares(u.data_ptr(), ws.data_ptr(), u[0].numel(), u.shape[0], _lib.stream_ptr(u.device))
    _lib.check(rc, "fsb_muon_sum_squares")
    count_launch()
    return ws


def _prepare(momentum, grad, mu, nesterov, count):
    """Momentum update in place and the bf16 direction before orthogonalisation, with the squared norms of its ``count``
    equal matrices."""
    _ensure()
    g = grad.contiguous()
    assert momentum.is_contiguous() and momentum.dtype == torch.float32 and momentum.shape == grad.shape
    n = g.numel() // count
    u = torch.empty(g.shape, dtype=torch.bfloat16, device=g.device)
    ws = _workspace(g.device, n, count)
    rc = _lib.load().fsb_muon_prepare(momentum.data_ptr(), g.data_ptr(), int(g.dtype == torch.float32), u.data_ptr(),
                                      ws.data_ptr(), n, count, mu, int(nesterov), _lib.stream_ptr(g.device))
    _lib.check(rc, "fsb_muon_prepare")
    count_launch()
    return u, ws


def muon_direction_(momentum: torch.Tensor, grad: torch.Tensor, mu: float, nesterov: bool, steps: int,
                    coeffs=NS_COEFFS, eps: float = 1e-7) -> torch.Tensor:
    """Momentum update (in place, fp32) + Nesterov + normalise + Newton-Schulz; returns the bf16
    direction with the shape of ``grad`` (2-D, or on CUDA a stack ``[n, rows, cols]`` of equal matrices that
    ``batched_ns_supported`` accepts)."""
    assert momentum.shape == grad.shape and (grad.dim() == 2 or batched_ns_supported(grad))
    if not grad.is_cuda:
        momentum.lerp_(grad.float(), 1 - mu)
        u = grad.float().lerp(momentum, mu) if nesterov else momentum
        return _newton_schulz_cpu(u, steps, coeffs, eps)
    count = grad.shape[0] if grad.dim() == 3 else 1
    u, ws = _prepare(momentum, grad, mu, nesterov, count)
    if grad.dim() == 3:
        return orthogonalise_stack_(u, steps, coeffs, eps, ws)
    return ns_iterations(_normalise_(u, ws, eps), steps, coeffs)


def orthogonalise_stack_(u: torch.Tensor, steps: int, coeffs, eps: float, ws: torch.Tensor | None = None) -> torch.Tensor:
    """Approximate polar factors of a contiguous bf16 stack that ``batched_ns_supported`` accepts; overwrites ``u``. What a
    stack that stays where it is stored (``ws``: the norms' workspace that its momentum kernel left) and matrices that
    came over an exchange have in common, so that the number of ranks does not show in the bits."""
    assert u.dtype == torch.bfloat16 and u.is_contiguous()
    return ns_iterations_batched(_normalise_(u, _sum_squares(u) if ws is None else ws, eps), steps, coeffs)


def muon_momentum_direction_(momentum: torch.Tensor, grad: torch.Tensor, mu: float, nesterov: bool) -> torch.Tensor:
    """``M <- lerp(M, g, 1-mu)`` in place (fp32) and return ``u = lerp(g, M, mu)`` (Nesterov) or ``M`` as bf16,
    in the shape of ``grad``: the elementwise half of a Muon step, for rows that are orthogonalised elsewhere."""
    assert momentum.shape == grad.shape and momentum.dtype == torch.float32
    if not grad.is_cuda:
        momentum.lerp_(grad.float(), 1 - mu)
        u = grad.float().lerp(momentum, mu) if nesterov else momentum
        return u.to(torch.bfloat16)
    return _prepare(momentum, grad, mu, nesterov, 1)[0]


def muon_apply_(param: torch.Tensor, direction: torch.Tensor, lr: float, weight_decay: float, ratio: float):
    """``p <- p (1 - lr*wd) - lr*ratio*direction`` in place."""
    if not param.is_cuda:
        param.mul_(1 - lr * weight_decay).add_(direction.to(param.dtype), alpha=-lr * ratio)
        return
    _ensure()
    assert param.is_contiguous() and direction.is_contiguous() and direction.dtype == torch.bfloat16
    rc = _lib.load().fsb_muon_update(param.data_ptr(), int(param.dtype == torch.float32), direction.data_ptr(),
                                     param.numel(), 1.0 - lr * weight_decay, lr * ratio,
                                     _lib.stream_ptr(param.device))
    _lib.check(rc, "fsb_muon_update")
    count_launch()
