"""Tensor-level entry points of the op library.

CUDA tensors go to the hand-written sm_100a kernels in ``libss_kernels.so``;
CPU tensors go to the plain-PyTorch definitions in :mod:`.reference`, which are
also the numerical oracles of the kernel tests. There is no third path: a CUDA
tensor with the library missing raises.
"""
from __future__ import annotations

import ctypes
import math

import os

import torch

from . import _lib, reference

_BF16 = torch.bfloat16


# SS_KERNELS=library is the comparison arm: the same planner, runtime and model code, but every op
# runs on vendor libraries and eager PyTorch (cuBLAS GEMMs, flash-attn, elementwise tensor
# operations) instead of this repository's kernels. It exists to be timed against, never as a
# fallback: nothing selects it but the variable.
_LIBRARY = os.environ.get("SS_KERNELS", "native") == "library"


def _cuda(t: torch.Tensor) -> bool:
    return t.is_cuda and not _LIBRARY


def _gemm_library(a, b, a_mn, b_mn, out, accumulate, alpha, out_dtype):
    """cuBLAS arm of ``gemm`` (bf16 operands, fp32 accumulation inside the library)."""
    am = a.t() if a_mn else a
    bm = b if b_mn else b.t()
    if out is None:
        res = torch.mm(am, bm)
        return (res if alpha == 1.0 else res * alpha).to(out_dtype)
    if out.dtype == am.dtype and out.is_contiguous():
        return torch.addmm(out, am, bm, beta=1.0 if accumulate else 0.0, alpha=alpha, out=out)
    res = torch.mm(am, bm).to(out.dtype)
    if alpha != 1.0:
        res = res * alpha
    return out.add_(res) if accumulate else out.copy_(res)


# Calls on the GPU go to the native module first, which takes operands that need nothing done to them and answers
# NotImplemented for all others (and until a device's status word exists): those go on in Python.
def _host(t: torch.Tensor):
    return _lib.host() if t.is_cuda and not _LIBRARY else None


def _ptr(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


# ------------------------------------------------------------------------ GEMM
# plain GEMMs of 256 x 128 and more enter at the CTA-pair kernel, which hands outputs of one wave of 128 x 128 tiles
# to the single-CTA kernel; SS_GEMM_PAIR=0 keeps all of them on that one
_PAIR_GEMM = os.environ.get("SS_GEMM_PAIR", "1") == "1"


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False,
         out: torch.Tensor | None = None, accumulate: bool = False, alpha: float = 1.0,
         out_dtype: torch.dtype | None = None, bn: int = 0) -> torch.Tensor:
    """``C[M,N] (+)= alpha * op(A) @ op(B)`` with bf16 operands, fp32 accumulation.

    ``a_mn``: A is stored ``[K, M]`` (else ``[M, K]``); ``b_mn``: B is stored
    ``[K, N]`` (else ``[N, K]``). ``accumulate`` adds the existing ``out``.
    """
    host = _host(a)
    if host is not None and _PAIR_GEMM and bn == 0 and (out is not None or out_dtype is None or out_dtype == _BF16):
        got = host.gemm(a, b, bool(a_mn), bool(b_mn), out, bool(accumulate), alpha)
        if got is not NotImplemented:
            return got
    M = a.shape[1] if a_mn else a.shape[0]
    K = a.shape[0] if a_mn else a.shape[1]
    N = b.shape[1] if b_mn else b.shape[0]
    Kb = b.shape[0] if b_mn else b.shape[1]
    if K != Kb:
        raise ValueError(f"contraction mismatch: {tuple(a.shape)} vs {tuple(b.shape)}")
    if out is None:
        if accumulate:
            raise ValueError("accumulate needs an existing output")
        out_dtype = out_dtype or a.dtype
    elif out.shape != (M, N):
        raise ValueError(f"output shape {tuple(out.shape)} != {(M, N)}")
    if a.is_cuda and _LIBRARY:
        return _gemm_library(a, b, a_mn, b_mn, out, accumulate, alpha, out_dtype or a.dtype)
    if not _cuda(a):
        return reference.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=accumulate,
                              alpha=alpha, out_dtype=out_dtype or a.dtype)
    if a.dtype != _BF16 or b.dtype != _BF16:
        raise TypeError("gemm operands must be bfloat16 on CUDA")
    lda, sa = a.stride()
    ldb, sb = b.stride()
    if sa != 1 or sb != 1:
        raise ValueError("gemm operands must have unit inner stride")
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    ldc, sc = out.stride()
    f32 = out.dtype == torch.float32
    if sc != 1 or not (f32 or out.dtype == _BF16):
        raise ValueError("gemm output must be bf16/fp32 with unit inner stride")
    if N % 8 or lda % 8 or ldb % 8 or ldc % (4 if f32 else 8):
        # TMA moves 16-byte pieces: say which size breaks that instead of returning the kernel's code
        raise ValueError(f"gemm on the GPU needs N and the row strides in multiples of 8 elements "
                         f"(N={N}, strides {lda}, {ldb}, {ldc}); pad the operand")
    if _PAIR_GEMM and bn == 0 and M >= 256 and N >= 128:
        # CTA-pair kernel (tcgen05 cta_group::2): 256x256 tiles, half the shared-memory
        # traffic per FLOP of the single-CTA kernel, which takes the outputs of one wave from there
        rc = _lib.lib().ss_gemm2_bf16(
            a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, lda, ldb, ldc, int(a_mn), int(b_mn), int(f32),
            int(accumulate), float(alpha), 0, _lib.status_ptr(a), _lib.stream_ptr())
        _lib.check(rc, "ss_gemm2_bf16")
        return out
    rc = _lib.lib().ss_gemm_bf16(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, lda, ldb, ldc, int(a_mn), int(b_mn), int(f32), int(accumulate),
        float(alpha), int(bn), 0, _lib.status_ptr(a), _lib.stream_ptr())
    _lib.check(rc, "ss_gemm_bf16")
    return out


# ------------------------------------------------------------------------ gather fused into the GEMM
class PendingGather:
    """A sharded weight whose all-gather has not happened yet: the first GEMM that consumes the
    full-weight buffer pulls the shards from the peers itself (``ss_gemm2_gather_bf16``)."""

    def __init__(self, full: torch.Tensor, shard_ptrs, per: int, world: int, rank: int, fallback):
        self.full, self.shard_ptrs, self.per, self.world, self.rank = full, shard_ptrs, per, world, rank
        self.fallback = fallback          # gathers with the stand-alone kernel instead


_pending_gathers: dict[int, PendingGather] = {}
fused_gather_launches = 0


def register_gather(info: PendingGather) -> None:
    _pending_gathers[info.full.data_ptr()] = info


def flush_gathers(ptrs=None) -> int:
    """Runs the stand-alone gather for every registered weight no GEMM consumed (all of them, or
    those whose buffers start at ``ptrs``). Returns how many there were."""
    keys = [k for k in list(_pending_gathers) if ptrs is None or k in ptrs]
    for k in keys:
        _pending_gathers.pop(k).fallback()
    return len(keys)


def _gemm_gather(x: torch.Tensor, info: PendingGather, out, accumulate: bool):
    global fused_gather_launches
    w = info.full
    N, K = w.shape
    M = x.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    counters = torch.zeros(-(-N // 256), dtype=torch.int32, device=x.device)
    import ctypes
    ptrs = (ctypes.c_void_p * info.world)(*info.shard_ptrs)
    rc = _lib.lib().ss_gemm2_gather_bf16(
        x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, x.stride(0), out.stride(0),
        int(out.dtype == torch.float32), int(accumulate), 1.0, ptrs, info.per, info.world, info.rank,
        counters.data_ptr(), 0, 0, _lib.status_ptr(x), _lib.stream_ptr())
    _lib.check(rc, "ss_gemm2_gather_bf16")
    fused_gather_launches += 1
    return out


def _plain_rows(*tensors) -> bool:
    """Are these 2-D bf16 CUDA tensors with rows that TMA and 16-byte stores can take?"""
    return all(t.is_cuda and t.dtype == _BF16 and t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0
               and t.shape[1] % 8 == 0 and t.data_ptr() % 16 == 0 for t in tensors)


def _fused_gemm(*tensors) -> bool:
    """Do these operands of a GEMM with more than a store in its epilogue run on the kernels of ``gemm`` as they are?"""
    return not _LIBRARY and not _pending_gathers and _PAIR_GEMM and _plain_rows(*tensors)


def linear_residual(x, w, residual, out=None):
    """``residual[T,N] + x[T,K] @ w[N,K]^T``; ``residual`` is only read (and may be ``out``)."""
    host = _host(x)
    if host is not None and _PAIR_GEMM and not _pending_gathers:
        got = host.linear_residual(x, w, residual, out)
        if got is not NotImplemented:
            return got
    if out is None:
        out = torch.empty_like(residual)
    M, N, K = x.shape[0], w.shape[0], x.shape[1]
    if not (_fused_gemm(x, w, residual, out) and w.shape[1] == K > 0 and out.shape == residual.shape == (M, N)):
        if out is not residual:
            out.copy_(residual)
        return linear_fwd(x, w, out=out, accumulate=True)
    _lib.check(_lib.lib().ss_gemm2_residual_bf16(
        x.data_ptr(), w.data_ptr(), residual.data_ptr(), out.data_ptr(), M, N, K, x.stride(0), w.stride(0),
        residual.stride(0), out.stride(0), _lib.status_ptr(x), _lib.stream_ptr()), "ss_gemm2_residual_bf16")
    return out


def swiglu_linear(x, w13, gu=None, out=None, keep_gu=True):
    """``gu = x @ w13^T`` (gate columns, then up columns) and ``h = silu(gate) * up`` by one kernel: ``(gu, h)``.
    Without ``keep_gu`` the projections are not written and the first is None."""
    host = _host(x)
    if host is not None and _PAIR_GEMM and not _pending_gathers:
        got = host.swiglu_linear(x, w13, gu, out, bool(keep_gu))
        if got is not NotImplemented:
            return got
    T, F2, K = x.shape[0], w13.shape[0], x.shape[1]
    keep_gu = keep_gu or gu is not None
    given = [t for t in (gu, out) if t is not None]
    if not (_fused_gemm(x, w13, *given) and w13.shape[1] == K and F2 % 16 == 0):
        gu = linear_fwd(x, w13, out=gu)
        return (gu if keep_gu else None), swiglu_fwd(gu, out=out)
    if keep_gu and gu is None:
        gu = torch.empty((T, F2), dtype=x.dtype, device=x.device)
    h = torch.empty((T, F2 // 2), dtype=x.dtype, device=x.device) if out is None else out
    _lib.check(_lib.lib().ss_gemm2_swiglu_bf16(
        x.data_ptr(), w13.data_ptr(), _ptr(gu), h.data_ptr(), T, F2 // 2, K, x.stride(0), w13.stride(0),
        0 if gu is None else gu.stride(0), h.stride(0), _lib.status_ptr(x), _lib.stream_ptr()), "ss_gemm2_swiglu_bf16")
    return gu, h


def swiglu_linear_dgrad(dy, w2, gu):
    """The gradient of ``gu`` for ``y = h @ w2^T`` with ``h = silu(gate) * up``: ``dy @ w2`` goes through SwiGLU's
    gradient where the products leave, and is never stored."""
    host = _host(dy)
    if host is not None and _PAIR_GEMM and not _pending_gathers:
        got = host.swiglu_linear_dgrad(dy, w2, gu)
        if got is not NotImplemented:
            return got
    T, F, K = dy.shape[0], w2.shape[1], dy.shape[1]
    if not (_fused_gemm(dy, w2, gu) and w2.shape[0] == K and gu.shape == (T, 2 * F)):
        return swiglu_bwd(gu, linear_dgrad(dy, w2))
    dgu = torch.empty((T, 2 * F), dtype=gu.dtype, device=gu.device)
    _lib.check(_lib.lib().ss_gemm2_swiglu_bwd_bf16(
        dy.data_ptr(), w2.data_ptr(), gu.data_ptr(), dgu.data_ptr(), T, F, K, dy.stride(0), w2.stride(0),
        gu.stride(0), dgu.stride(0), _lib.status_ptr(dy), _lib.stream_ptr()), "ss_gemm2_swiglu_bwd_bf16")
    return dgu


def linear_fwd(x, w, out=None, accumulate=False):
    """``y[T,N] (+)= x[T,K] @ w[N,K]^T``. A weight registered by ``register_gather`` is gathered
    from its shards by this GEMM itself."""
    if _pending_gathers:
        info = _pending_gathers.pop(w.data_ptr(), None)
        if info is not None:
            fits = (_cuda(x) and x.dtype == _BF16 and w.dim() == 2 and w.is_contiguous() and x.stride(-1) == 1
                    and x.shape[0] >= 256 and w.shape[1] % 64 == 0 and w.shape[0] % 8 == 0
                    and (out is None or out.stride(-1) == 1))
            if fits:
                return _gemm_gather(x, info, out, accumulate)
            info.fallback()
    return gemm(x, w, out=out, accumulate=accumulate)


def linear_dgrad(dy, w, out=None, accumulate=False):
    """``dx[T,K] (+)= dy[T,N] @ w[N,K]``"""
    return gemm(dy, w, b_mn=True, out=out, accumulate=accumulate)


def linear_wgrad(dy, x, out=None, accumulate=False, out_dtype=None):
    """``dw[N,K] (+)= dy[T,N]^T @ x[T,K]`` -- the in-place gradient accumulation
    (reference: shadowspill::accumulate_matmul_)."""
    return gemm(dy, x, a_mn=True, b_mn=True, out=out, accumulate=accumulate, out_dtype=out_dtype)


# ------------------------------------------------------------------------ norms
def rmsnorm_fwd(x, w, eps=1e-5, zero_centered=False, delta=None, out=None, rstd=None):
    """``x += delta`` (optional, in place) then RMSNorm. Returns ``(y, rstd)``."""
    if not _cuda(x):
        y, rs = reference.rmsnorm_fwd(x, w, eps, zero_centered, delta)
        if out is not None:
            y = out.copy_(y)
        if rstd is not None:
            rs = rstd.copy_(rs)
        return y, rs
    got = _lib.host().rmsnorm_fwd(x, w, eps, bool(zero_centered), delta, out, rstd)
    if got is not NotImplemented:
        return got
    T, D = x.shape
    y = torch.empty_like(x) if out is None else out
    rs = torch.empty(T, dtype=torch.float32, device=x.device) if rstd is None else rstd
    rc = _lib.lib().ss_rmsnorm_fwd(x.data_ptr(), _ptr(delta), w.data_ptr(), y.data_ptr(),
                                   rs.data_ptr(), T, D, float(eps), int(zero_centered),
                                   _lib.status_ptr(x), _lib.stream_ptr())
    _lib.check(rc, "ss_rmsnorm_fwd")
    return y, rs


def rmsnorm_bwd(x, w, gy, rstd, dw, zero_centered=False, dx=None, accumulate=False):
    """Returns ``dx`` (added into ``dx`` when ``accumulate``); ``dw`` (fp32) is
    accumulated in place."""
    if not _cuda(x):
        dxr, dwr = reference.rmsnorm_bwd(x, w, gy, rstd, zero_centered)
        if dw is not None:
            dw.add_(dwr.to(dw.dtype))
        if dx is None:
            return dxr.to(x.dtype)
        dx.copy_(((dx.float() if accumulate else 0) + dxr).to(dx.dtype))
        return dx
    got = _lib.host().rmsnorm_bwd(x, w, gy, rstd, dw, bool(zero_centered), dx, bool(accumulate))
    if got is not NotImplemented:
        return got
    T, D = x.shape
    if dx is None:
        if accumulate:
            raise ValueError("accumulate needs dx")
        dx = torch.empty_like(x)
    if dw is not None and dw.dtype != torch.float32:
        raise TypeError("rmsnorm dw accumulator must be fp32")
    rc = _lib.lib().ss_rmsnorm_bwd(x.data_ptr(), w.data_ptr(), gy.data_ptr(), rstd.data_ptr(),
                                   dx.data_ptr(), _ptr(dw), T, D, int(zero_centered),
                                   int(accumulate), _lib.status_ptr(x), _lib.stream_ptr())
    _lib.check(rc, "ss_rmsnorm_bwd")
    return dx


def _heads_in_place(dh, *tensors) -> bool:
    """Can the strided head kernels read and write these views? They move 16-byte pieces and keep a head
    in at most two of them per lane; other views are copied to contiguous rows."""
    return dh % 8 == 0 and dh <= 512 and all(
        t is None or (_cuda(t) and t.dtype == _BF16 and t.stride(1) == 1 and t.stride(0) % 8 == 0
                      and t.data_ptr() % 16 == 0) for t in tensors)


def head_norm_(buf, w, heads, eps=1e-5, zero_centered=False, raw=None):
    """RMSNorm of each of the ``heads`` adjacent heads in the rows of ``buf`` (``[T, heads * dh]``, a view
    with unit inner stride), in place; ``raw`` (same shape) receives the input. Returns ``rstd``
    ``[T * heads]``."""
    T, dh = buf.shape[0], buf.shape[1] // heads
    if not _heads_in_place(dh, buf, raw):
        if raw is not None:
            raw.copy_(buf)
        y, rs = rmsnorm_fwd(buf.reshape(T * heads, dh), w, eps, zero_centered)
        buf.copy_(y.view(T, heads * dh))
        return rs
    rs = torch.empty(T * heads, dtype=torch.float32, device=buf.device)
    _lib.check(_lib.lib().ss_headnorm_fwd(
        buf.data_ptr(), buf.stride(0), w.data_ptr(), buf.data_ptr(), buf.stride(0), _ptr(raw),
        0 if raw is None else raw.stride(0), rs.data_ptr(), T, heads, dh, float(eps), int(zero_centered),
        _lib.stream_ptr()), "ss_headnorm_fwd")
    return rs


def head_norm_bwd_(raw, w, dbuf, rstd, dw, heads, zero_centered=False):
    """Rewrites ``dbuf`` (``[T, heads * dh]``, a view) with the gradient of :func:`head_norm_`'s input
    ``raw``; ``dw`` (fp32) is accumulated in place."""
    T, dh = dbuf.shape[0], dbuf.shape[1] // heads
    if not _heads_in_place(dh, dbuf, raw):
        dx = rmsnorm_bwd(raw.reshape(T * heads, dh), w, dbuf.reshape(T * heads, dh), rstd, dw, zero_centered)
        return dbuf.copy_(dx.view(T, heads * dh))
    if dw is not None and dw.dtype != torch.float32:
        raise TypeError("rmsnorm dw accumulator must be fp32")
    _lib.check(_lib.lib().ss_headnorm_bwd(
        raw.data_ptr(), raw.stride(0), w.data_ptr(), dbuf.data_ptr(), dbuf.stride(0), rstd.data_ptr(),
        dbuf.data_ptr(), dbuf.stride(0), _ptr(dw), T, heads, dh, int(zero_centered), _lib.stream_ptr()),
        "ss_headnorm_bwd")
    return dbuf


# ------------------------------------------------------------------------ rotary
def rope_(buf, positions, *, col0, heads, dh, rot=None, theta=10000.0, inverse=False):
    """In-place rotary on ``heads`` heads of width ``dh`` starting at column ``col0``
    of the 2-D buffer ``buf``; ``inverse`` applies the backward rotation."""
    rot = dh if rot is None else rot
    if not _cuda(buf):
        return reference.rope_(buf, positions, col0, heads, dh, rot, theta, inverse)
    got = _lib.host().rope(buf, positions, col0, heads, dh, rot, theta, bool(inverse))
    if got is not NotImplemented:
        return got
    if positions.dtype != torch.int32:
        raise TypeError("positions must be int32")
    rc = _lib.lib().ss_rope(buf.data_ptr(), positions.data_ptr(), buf.shape[0], buf.stride(0),
                            col0, heads, dh, rot, float(theta), int(inverse), _lib.stream_ptr())
    _lib.check(rc, "ss_rope")
    return buf


# ------------------------------------------------------------------------ SwiGLU
def swiglu_fwd(gu, out=None):
    if not _cuda(gu):
        res = reference.swiglu_fwd(gu)
        return res if out is None else out.copy_(res)
    T, F2 = gu.shape
    h = torch.empty((T, F2 // 2), dtype=gu.dtype, device=gu.device) if out is None else out
    _lib.check(_lib.lib().ss_swiglu_fwd(gu.data_ptr(), h.data_ptr(), T, F2 // 2,
                                        _lib.stream_ptr()), "ss_swiglu_fwd")
    return h


def swiglu_bwd(gu, dh, out=None):
    if not _cuda(gu):
        res = reference.swiglu_bwd(gu, dh)
        return res if out is None else out.copy_(res)
    T, F2 = gu.shape
    dgu = torch.empty_like(gu) if out is None else out
    _lib.check(_lib.lib().ss_swiglu_bwd(gu.data_ptr(), dh.data_ptr(), dgu.data_ptr(), T, F2 // 2,
                                        _lib.stream_ptr()), "ss_swiglu_bwd")
    return dgu


# ------------------------------------------------------------------------ embedding
def embedding_fwd(ids, W, out=None):
    if not _cuda(W):
        res = reference.embedding_fwd(ids, W)
        return res if out is None else out.copy_(res)
    T = ids.numel()
    V, D = W.shape
    o = torch.empty((T, D), dtype=W.dtype, device=W.device) if out is None else out
    _lib.check(_lib.lib().ss_embedding_fwd(ids.data_ptr(), W.data_ptr(), o.data_ptr(), T, D, V,
                                           _lib.stream_ptr()), "ss_embedding_fwd")
    return o


def embedding_bwd(ids, g, dW):
    """``dW[ids[t]] += g[t]`` (dW fp32 or bf16)."""
    if not _cuda(g):
        return reference.embedding_bwd(ids, g, dW)
    T = ids.numel()
    V, D = dW.shape
    _lib.check(_lib.lib().ss_embedding_bwd(ids.data_ptr(), g.data_ptr(), dW.data_ptr(), T, D, V,
                                           int(dW.dtype == torch.float32), _lib.stream_ptr()),
               "ss_embedding_bwd")
    return dW


# ------------------------------------------------------------------------ cross-entropy block
def cross_entropy_(logits, targets, weights, loss_sum, *, grad_scale=1.0, write_grad=True,
                   lse=None):
    """Adds the weighted loss of a logits block into ``loss_sum`` (fp32[1]) and
    rewrites ``logits`` with its gradient. Masked rows carry weight 0."""
    if not _cuda(logits):
        loss, _ = reference.cross_entropy_(logits, targets, weights, grad_scale, write_grad)
        loss_sum.add_(loss)
        return loss_sum
    R, V = logits.shape
    _lib.check(_lib.lib().ss_cross_entropy(logits.data_ptr(), targets.data_ptr(), _ptr(weights),
                                           loss_sum.data_ptr(), _ptr(lse), R, V, logits.stride(0),
                                           float(grad_scale), int(write_grad), _lib.stream_ptr()),
               "ss_cross_entropy")
    return loss_sum


def clipped_policy_(logits, targets, weights, old_logp, advantage, loss_sum, *, clip=0.2,
                    ref_logp=None, ref_beta=0.0, grad_scale=1.0, write_grad=True, logp=None):
    """Clipped policy objective on a logits block: adds the weighted loss into
    ``loss_sum`` and rewrites ``logits`` with its gradient; ``logp`` (fp32[R]) receives
    the target log-probabilities."""
    if not _cuda(logits):
        loss, lp = reference.clipped_policy_(logits, targets, weights, old_logp, advantage, clip,
                                             ref_logp, ref_beta, grad_scale, write_grad)
        loss_sum.add_(loss)
        if logp is not None:
            logp.copy_(lp)
        return loss_sum
    R, V = logits.shape
    _lib.check(_lib.lib().ss_token_objective(
        logits.data_ptr(), targets.data_ptr(), _ptr(weights), loss_sum.data_ptr(), _ptr(logp), R, V,
        logits.stride(0), float(grad_scale), int(write_grad), 1, old_logp.data_ptr(),
        advantage.data_ptr(), float(clip), _ptr(ref_logp), float(ref_beta), _lib.stream_ptr()),
        "ss_token_objective")
    return loss_sum


def target_logprobs_(logits, targets, logp):
    """log p(target) per row of a logits block into ``logp`` (fp32[R]); logits unchanged."""
    if not _cuda(logits):
        lf = logits.float()
        V = logits.shape[-1]
        picked = lf.gather(1, targets.clamp(0, V - 1)[:, None])[:, 0]
        logp.copy_(picked - torch.logsumexp(lf, dim=-1))
        return logp
    R, V = logits.shape
    scratch = torch.zeros(1, dtype=torch.float32, device=logits.device)
    _lib.check(_lib.lib().ss_token_objective(
        logits.data_ptr(), targets.data_ptr(), None, scratch.data_ptr(), logp.data_ptr(), R, V,
        logits.stride(0), 1.0, 0, 0, None, None, 0.0, None, 0.0, _lib.stream_ptr()),
        "ss_token_objective")
    return logp


# ------------------------------------------------------------------------ AdamW
def adamw_(p, g, m, v, *, lr, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.0, step=1,
           grad_scale=1.0, seed=0, offset=0, stochastic_param=True, stochastic_state=True):
    """Fused AdamW on flat tensors. bf16 parameters/moments use stochastic
    rounding driven by a counter RNG keyed on (seed, step, global element index),
    so a shard updated alone produces the same bits as the whole tensor."""
    if not _cuda(p):
        return reference.adamw_(p, g, m, v, lr=lr, beta1=beta1, beta2=beta2, eps=eps,
                                weight_decay=weight_decay, step=step, grad_scale=grad_scale)
    n = p.numel()
    L = _lib.lib()
    if p.dtype == torch.float32:
        _lib.check(L.ss_adamw_f32(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), n,
                                  lr, beta1, beta2, eps, weight_decay, step, grad_scale,
                                  _lib.stream_ptr()), "ss_adamw_f32")
        return
    _lib.check(L.ss_adamw_sr(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), n,
                             int(g.dtype == torch.float32), lr, beta1, beta2, eps, weight_decay,
                             step, grad_scale, seed, offset, int(stochastic_param),
                             int(stochastic_state), _lib.stream_ptr()), "ss_adamw_sr")


ADAMW_MANY_ELEMENTS = 148 * 2 * 256 * 8     # as the kernel's launcher has it, which refuses larger ones


def adamw_many_(tensors, *, lr, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.0, step=1, grad_scale=1.0,
                seed=0, stochastic_param=True, stochastic_state=True):
    """``adamw_`` for every ``(p, g, m, v, offset)`` of flat tensors, with the same bits. Small bf16
    tensors share a launch: one by one they cost their launches (27 of a small model: 0.3 ms)."""
    hyper = dict(lr=lr, beta1=beta1, beta2=beta2, eps=eps, weight_decay=weight_decay, step=step,
                 grad_scale=grad_scale, seed=seed, stochastic_param=stochastic_param,
                 stochastic_state=stochastic_state)
    table, seen = [], set()
    for p, g, m, v, offset in tensors:
        n, at = p.numel(), p.data_ptr()
        # a parameter listed twice is updated twice, in order
        if not _cuda(p) or p.dtype != _BF16 or n > ADAMW_MANY_ELEMENTS or at in seen:
            if at in seen and table:
                _adamw_table(table, hyper)
                table, seen = [], set()
            adamw_(p, g, m, v, offset=offset, **hyper)
            continue
        seen.add(at)
        table += (at, g.data_ptr(), m.data_ptr(), v.data_ptr(), n, offset, int(g.dtype == torch.float32))
    if table:
        _adamw_table(table, hyper)


def _adamw_table(table, h):
    k = len(table) // 7
    _lib.check(_lib.lib().ss_adamw_sr_many(
        (ctypes.c_longlong * len(table))(*table), k, h["lr"], h["beta1"], h["beta2"], h["eps"], h["weight_decay"],
        h["step"], h["grad_scale"], h["seed"], int(h["stochastic_param"]), int(h["stochastic_state"]),
        _lib.stream_ptr()), "ss_adamw_sr_many")


def sumsq(x, partials, out, accumulate=False):
    """Sum of squares into ``out`` (fp32[1]) using caller-owned ``partials`` (fp32[256])."""
    if not _cuda(x):
        val = x.float().square().sum()
        out.copy_(out + val if accumulate else val.reshape(1))
        return out
    _lib.check(_lib.lib().ss_sumsq(x.data_ptr(), x.numel(), partials.data_ptr(), out.data_ptr(),
                                   int(accumulate), _lib.stream_ptr()), "ss_sumsq")
    return out


# ------------------------------------------------------------------------ attention
def attention_varlen(q, k, v, cu_seqlens, max_seqlen, scale=None, out=None, lse=None):
    """Packed causal GQA forward. Returns ``(out, lse)``; ``lse`` is fp32 ``[Hq, T]``."""
    if not q.is_cuda:
        o, l = reference.attention_varlen(q, k, v, cu_seqlens, scale)
        if out is not None:
            o = out.copy_(o)
        if lse is not None:
            l = lse.copy_(l)
        return o, l
    from . import attention
    return attention.forward(q, k, v, cu_seqlens, max_seqlen, scale, out=out, lse=lse)


def attention_varlen_bwd(q, k, v, out, lse, dout, cu_seqlens, max_seqlen, scale=None):
    if not q.is_cuda:
        return reference.attention_varlen_bwd(q, k, v, out, lse, dout, cu_seqlens, scale)
    from . import attention
    return attention.backward(q, k, v, out, lse, dout, cu_seqlens, max_seqlen, scale)


def default_scale(dh: int) -> float:
    return 1.0 / math.sqrt(dh)
