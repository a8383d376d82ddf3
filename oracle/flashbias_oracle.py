"""CPU restatement of the FlashBias attention path.  TEST INFRASTRUCTURE ONLY.

This module is the oracle for the CUDA kernels: only the test-suite, the smoke
entry and the benchmark's CPU-baseline leg may import it.  Nothing in the
product package routes through it.

It restates, in plain PyTorch CPU ops, the naive attention the reference uses as
its own correctness baseline, and the gradient formulas of the reference's
backward kernel:

* forward      -- ``attention_torch`` (flash_bias/attention_func.py:16-55) with the
  dense bias materialised from the factors as ``q_bias @ k_bias^T``
  (flash_bias/benchmark.py:42-43); logits are
  ``softmax_scale * (q . k) + (q_bias . k_bias) [+ mask]`` with the bias NOT scaled
  (flash_bias/flash_bias_triton.py:246-256), causal masking is top-left aligned
  ``row >= col`` (:262), the additive mask comes after the bias (:263-282), and the
  log-sum-exp is natural-log (:321-323).
* backward     -- ``delta = rowsum(o * do)`` (:384-400), ``p = exp(s - lse)`` (:669-670),
  ``dv = p^T do`` (:697), ``dp = do v^T``, ``ds = p * (dp - delta)`` (:704-714),
  ``dk = scale * ds^T q`` (:717), ``dk_bias = ds^T q_bias`` (:719),
  ``dq = scale * ds k`` (:728), ``dq_bias = ds k_bias`` (:732).

Parity pin: the functions here are checked against outputs of the reference's own
``attention_torch`` + autograd, generated by ``tests/golden/make_golden.py`` in a
container that has the reference checked out, and committed under ``tests/golden``.

Deliberate choices where the reference leaves behaviour open:
* gradients of factors that are broadcast over batch and/or heads are summed over
  the broadcast dimensions (what autograd of the naive path gives);
* a query row with no visible key yields output 0 and lse = -inf (the naive path
  gives NaN there).
"""
from __future__ import annotations

import math
from typing import Optional, Tuple

import torch

__all__ = [
    "default_scale",
    "attention_forward",
    "attention_backward",
    "attention_forward_backward",
    "dense_bias",
]


def default_scale(softmax_scale, d: int) -> float:
    """``softmax_scale or 1/sqrt(d)`` (flash_bias/flash_bias_triton.py:1110)."""
    return float(softmax_scale) if softmax_scale else 1.0 / math.sqrt(d)


def _bh(x: torch.Tensor, b: int, h: int) -> torch.Tensor:
    """Slice (B|1, S, H|1, C) -> (S, C) for batch b and head h, honouring broadcast."""
    bb = b if x.shape[0] > 1 else 0
    hh = h if x.shape[2] > 1 else 0
    return x[bb, :, hh, :]


def _mask_bh(mask: torch.Tensor, b: int, h: int) -> torch.Tensor:
    """Slice (B|1, H|1, 1|Sq, Sk) -> (1|Sq, Sk)."""
    bb = b if mask.shape[0] > 1 else 0
    hh = h if mask.shape[1] > 1 else 0
    return mask[bb, hh]


def dense_bias(q_bias: torch.Tensor, k_bias: torch.Tensor) -> torch.Tensor:
    """(B|1,H|1,Sq,Sk) bias from (B|1,Sq,H|1,R) x (B|1,Sk,H|1,R) factors (benchmark.py:42-43)."""
    return torch.einsum("bqhr,bkhr->bhqk", q_bias, k_bias)


def _logits(q, k, qb, kb, mask2d, causal, scale, row0):
    s = (q @ k.transpose(0, 1)) * scale
    if qb is not None:
        s = s + qb @ kb.transpose(0, 1)
    if mask2d is not None:
        s = s + mask2d
    if causal:
        rows = torch.arange(row0, row0 + q.shape[0]).unsqueeze(1)
        cols = torch.arange(k.shape[0]).unsqueeze(0)
        s = s.masked_fill(cols > rows, float("-inf"))
    return s


def attention_forward(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    q_bias: Optional[torch.Tensor] = None,
    k_bias: Optional[torch.Tensor] = None,
    mask: Optional[torch.Tensor] = None,
    causal: bool = False,
    softmax_scale: Optional[float] = None,
    *,
    dtype: torch.dtype = torch.float32,
    block_rows: int = 4096,
    round_p: Optional[torch.dtype] = None,
) -> Tuple[torch.Tensor, torch.Tensor]:
    """Naive attention forward.  Returns (o (B,Sq,H,D), lse (B,H,Sq)) in ``dtype``.

    Works per (batch, head) and per block of query rows so that S = 32768 fits in
    host memory; softmax is row-wise, so the blocking does not change the arithmetic.

    ``round_p``: round the probabilities to that 16-bit type before ``p @ v``, as the reference kernel does
    (flash_bias/flash_bias_triton.py:317); used to measure what that mandated rounding alone costs.
    """
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    scale = default_scale(softmax_scale, D)
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    if q_bias is not None:
        q_bias, k_bias = q_bias.to(dtype), k_bias.to(dtype)
    if mask is not None:
        mask = mask.to(dtype)
    o = torch.empty(B, Sq, H, D, dtype=dtype)
    lse = torch.empty(B, H, Sq, dtype=dtype)
    for b in range(B):
        for h in range(H):
            kk, vv = k[b, :, h], v[b, :, h]
            kb = _bh(k_bias, b, h) if k_bias is not None else None
            m2 = _mask_bh(mask, b, h) if mask is not None else None
            for r0 in range(0, Sq, block_rows):
                r1 = min(Sq, r0 + block_rows)
                qb = _bh(q_bias, b, h)[r0:r1] if q_bias is not None else None
                mm = None
                if m2 is not None:
                    mm = m2 if m2.shape[0] == 1 else m2[r0:r1]
                s = _logits(q[b, r0:r1, h], kk, qb, kb, mm, causal, scale, r0)
                l = torch.logsumexp(s, dim=-1)
                p = torch.exp(s - torch.where(torch.isinf(l), torch.zeros_like(l), l).unsqueeze(1))
                p = torch.where(torch.isinf(l).unsqueeze(1), torch.zeros_like(p), p)
                if round_p is not None:
                    p = p.to(round_p).to(dtype)
                o[b, r0:r1, h] = p @ vv
                lse[b, h, r0:r1] = l
    return o, lse


def attention_backward(
    do: torch.Tensor,
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    o: torch.Tensor,
    lse: torch.Tensor,
    q_bias: Optional[torch.Tensor] = None,
    k_bias: Optional[torch.Tensor] = None,
    mask: Optional[torch.Tensor] = None,
    causal: bool = False,
    softmax_scale: Optional[float] = None,
    *,
    dtype: torch.dtype = torch.float32,
    block_rows: int = 4096,
    round_p: Optional[torch.dtype] = None,
):
    """Gradients (dq, dk, dv, dq_bias, dk_bias) from the reference's backward formulas.

    Factor gradients have the shape of the factors as given (broadcast dims summed).

    ``round_p``: round P (before ``p^T do``) and dS (before its four products) to that 16-bit type, as the
    reference kernel does (flash_bias/flash_bias_triton.py:696, :714).
    """
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    scale = default_scale(softmax_scale, D)
    do, q, k, v, o, lse = (t.to(dtype) for t in (do, q, k, v, o, lse))
    has_bias = q_bias is not None
    if has_bias:
        q_bias, k_bias = q_bias.to(dtype), k_bias.to(dtype)
    if mask is not None:
        mask = mask.to(dtype)
    dq = torch.zeros_like(q)
    dk = torch.zeros_like(k)
    dv = torch.zeros_like(v)
    dqb = torch.zeros_like(q_bias) if has_bias else None
    dkb = torch.zeros_like(k_bias) if has_bias else None
    for b in range(B):
        for h in range(H):
            kk, vv = k[b, :, h], v[b, :, h]
            kb = _bh(k_bias, b, h) if has_bias else None
            m2 = _mask_bh(mask, b, h) if mask is not None else None
            for r0 in range(0, Sq, block_rows):
                r1 = min(Sq, r0 + block_rows)
                qq = q[b, r0:r1, h]
                qb = _bh(q_bias, b, h)[r0:r1] if has_bias else None
                mm = None
                if m2 is not None:
                    mm = m2 if m2.shape[0] == 1 else m2[r0:r1]
                s = _logits(qq, kk, qb, kb, mm, causal, scale, r0)
                l = lse[b, h, r0:r1]
                dead = torch.isinf(l)
                p = torch.exp(s - torch.where(dead, torch.zeros_like(l), l).unsqueeze(1))
                p = torch.where(dead.unsqueeze(1), torch.zeros_like(p), p)
                dd = do[b, r0:r1, h]
                delta = (o[b, r0:r1, h] * dd).sum(-1, keepdim=True)
                ds = p * (dd @ vv.transpose(0, 1) - delta)
                if round_p is not None:
                    p = p.to(round_p).to(dtype)
                    ds = ds.to(round_p).to(dtype)
                dv[b, :, h] += p.transpose(0, 1) @ dd
                dq[b, r0:r1, h] = (ds @ kk) * scale
                dk[b, :, h] += (ds.transpose(0, 1) @ qq) * scale
                if has_bias:
                    bq = b if q_bias.shape[0] > 1 else 0
                    hq = h if q_bias.shape[2] > 1 else 0
                    bk = b if k_bias.shape[0] > 1 else 0
                    hk = h if k_bias.shape[2] > 1 else 0
                    dqb[bq, r0:r1, hq] += ds @ kb
                    dkb[bk, :, hk] += ds.transpose(0, 1) @ qb
    return dq, dk, dv, dqb, dkb


def attention_forward_backward(q, k, v, q_bias, k_bias, mask, causal, softmax_scale, do,
                               *, dtype=torch.float32, block_rows: int = 4096):
    """Convenience: forward then backward with an explicit dO. Returns (o, lse, grads)."""
    o, lse = attention_forward(q, k, v, q_bias, k_bias, mask, causal, softmax_scale,
                               dtype=dtype, block_rows=block_rows)
    grads = attention_backward(do, q, k, v, o, lse, q_bias, k_bias, mask, causal, softmax_scale,
                               dtype=dtype, block_rows=block_rows)
    return o, lse, grads
