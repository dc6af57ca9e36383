"""The output head over the rows that its loss scores.

The gradient of a logits row whose token carries no loss (no target, or weight 0) is zero and nothing else of the row
is used, so neither its logits nor its share of the two gradients needs to be formed. ``scored(...)`` returns the rows
the head works on: those tokens' hidden states in order, counted on the device (nothing is read back; blocks past the
count run their kernels on no rows), or all rows as they are where finding them would not pay. The reference evaluates
every row and multiplies by the weight (packages/workloads/src/shadowspill_workloads/models/shared/token_head.py:63-68).
"""
from __future__ import annotations

import torch

from . import _lib
from . import functional as F

_P, _I, _L, _F = _lib.c_p, _lib.c_int, _lib.c_ll, _lib.c_f
_lib.register("ss_scored_rows", [_P, _P, _I, _I, _P, _P, _P, _P])
_lib.register("ss_take_rows", [_P, _L, _P, _P, _L, _I, _I, _P])
_lib.register("ss_gemm2_rows_bf16", [_P, _P, _P, _I, _I, _I, _L, _L, _L, _I, _I, _I, _P, _I, _P, _P])
_lib.register("ss_token_objective_rows", [_P, _P, _P, _P, _P, _I, _P, _I, _I, _L, _F, _I, _I, _P, _P, _F, _P, _F, _P])

# Multiply-adds of one product over all rows from which the rows are worth finding: a head whose rows are all scored
# pays for the three small kernels and gains nothing, so the line lies where that is 2 % at most. All rows -> scored rows,
# us, both in turn, for all / nine in ten / half of them scored:
#   512 rows, 50,304 x 2,048 (5e10): 348 -> 376, 347 -> 375, 341 -> 323;  1,000 rows (1e11): 488 -> 503, 491 -> 502, 551 -> 435
#   1,000 rows, 128,256 x 2,048 (2.6e11): 1408 -> 1436, 1453 -> 1454, 1461 -> 1058
#   1,000 rows, 151,936 x 2,048 (3.1e11): 1508 -> 1532, 1805 -> 1790, 1762 -> 1276
#   1,000 rows, 128,256 x 4,096 (5.3e11): 2405 -> 2427, 2792 -> 2741, 2499 -> 1801;  8,192 rows: 21190 -> 21260, .., 19860 -> 10300
# Below the line half-masked heads go without what they could gain.
MIN_WORK = 3e11


class AllRows:
    """Every row, as it is."""

    def take(self, h):
        return h

    def put(self, dh):
        return dh

    def logits(self, h, W, r0, r1):
        return F.linear_fwd(h[r0:r1], W)

    def cross_entropy_(self, logits, targets, weights, loss_sum, r0, r1, **kw):
        F.cross_entropy_(logits, targets[r0:r1], weights[r0:r1], loss_sum, **kw)

    def clipped_policy_(self, logits, targets, weights, old_logp, advantage, loss_sum, r0, r1, ref_logp=None, **kw):
        F.clipped_policy_(logits, targets[r0:r1], weights[r0:r1], old_logp[r0:r1], advantage[r0:r1], loss_sum,
                          ref_logp=None if ref_logp is None else ref_logp[r0:r1], **kw)

    def wgrad(self, dlogits, h, out, accumulate, r0, r1):
        F.linear_wgrad(dlogits, h[r0:r1], out=out, accumulate=accumulate)

    def dgrad(self, dlogits, W, dh, r0, r1):
        F.linear_dgrad(dlogits, W, out=dh[r0:r1])


class ScoredRows:
    """The scored rows in order; row blocks ``[r0, r1)`` below count in them."""

    def __init__(self, h, W, targets, weights):
        T = h.shape[0]
        self.T, self.V = T, W.shape[0]
        self.rows, self.slot = torch.empty((2, T), dtype=torch.int32, device=h.device)
        self.count = torch.empty(1, dtype=torch.int32, device=h.device)
        _lib.check(_lib.lib().ss_scored_rows(targets.data_ptr(), weights.data_ptr(), T, self.V, self.rows.data_ptr(),
                                             self.slot.data_ptr(), self.count.data_ptr(), _lib.stream_ptr()),
                   "ss_scored_rows")

    def _select(self, x, index):
        out = torch.empty_like(x)
        _lib.check(_lib.lib().ss_take_rows(x.data_ptr(), x.stride(0), index.data_ptr(), out.data_ptr(), out.stride(0),
                                           self.T, x.shape[1], _lib.stream_ptr()), "ss_take_rows")
        return out

    def take(self, h):
        """The scored rows of ``h``, zero rows behind them."""
        return self._select(h, self.rows)

    def put(self, dh):
        """Gradients of the scored rows back to their tokens, zero for the others."""
        return self._select(dh, self.slot)

    def _gemm(self, a, b, out, M, N, K, a_mn, b_mn, accumulate, r0):
        _lib.check(_lib.lib().ss_gemm2_rows_bf16(
            a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn,
            int(accumulate), self.count.data_ptr(), r0, _lib.status_ptr(a), _lib.stream_ptr()), "ss_gemm2_rows_bf16")
        return out

    def logits(self, h, W, r0, r1):
        out = torch.empty((r1 - r0, self.V), dtype=h.dtype, device=h.device)
        return self._gemm(h[r0:r1], W, out, r1 - r0, self.V, h.shape[1], 0, 0, False, r0)

    def _objective(self, logits, targets, weights, loss_sum, r0, mode, old, adv, clip, ref, beta, grad_scale, write_grad):
        R, V = logits.shape
        _lib.check(_lib.lib().ss_token_objective_rows(
            logits.data_ptr(), targets.data_ptr(), weights.data_ptr(), self.rows.data_ptr(), self.count.data_ptr(), r0,
            loss_sum.data_ptr(), R, V, logits.stride(0), float(grad_scale), int(write_grad), mode, F._ptr(old),
            F._ptr(adv), float(clip), F._ptr(ref), float(beta), _lib.stream_ptr()), "ss_token_objective_rows")

    def cross_entropy_(self, logits, targets, weights, loss_sum, r0, r1, grad_scale=1.0, write_grad=True):
        self._objective(logits, targets, weights, loss_sum, r0, 0, None, None, 0.0, None, 0.0, grad_scale, write_grad)

    def clipped_policy_(self, logits, targets, weights, old_logp, advantage, loss_sum, r0, r1, clip=0.2, ref_logp=None,
                        ref_beta=0.0, grad_scale=1.0, write_grad=True):
        self._objective(logits, targets, weights, loss_sum, r0, 1, old_logp, advantage, clip, ref_logp, ref_beta,
                        grad_scale, write_grad)

    def wgrad(self, dlogits, h, out, accumulate, r0, r1):
        self._gemm(dlogits, h[r0:r1], out, self.V, h.shape[1], r1 - r0, 1, 1, accumulate, r0)

    def dgrad(self, dlogits, W, dh, r0, r1):
        self._gemm(dlogits, W, dh[r0:r1], r1 - r0, W.shape[1], self.V, 0, 1, False, r0)


def scored(h, W, targets, weights, Gw=None):
    """The rows of ``h`` [T,D] that a head with matrix ``W`` [V,D] (gradient ``Gw``) works on."""
    tensors = [t for t in (h, W, Gw) if t is not None]
    if (float(h.shape[0]) * W.shape[0] * W.shape[1] < MIN_WORK or not F._fused_gemm(*tensors) or W.shape[0] % 8
            or weights.dtype != torch.float32 or targets.dtype != torch.int64
            or not (targets.is_contiguous() and weights.is_contiguous())):
        return AllRows()
    return ScoredRows(h, W, targets, weights)
