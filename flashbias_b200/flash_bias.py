"""``flash_bias_func`` -- the reference's operator on top of the B200 C ABI.

Mirrors ``FlashBiasFunc`` / ``flash_bias_func`` of the reference
(flash_bias/flash_bias_triton.py:1345-1405): same positional signature
``(q, k, v, q_bias=None, k_bias=None, mask=None, causal=False, softmax_scale=None)``, same layouts
((B, S, H, D) tensors, (B|1, S, H|1, R) factors, 4-D additive mask), same host-side checks and
messages (:1102-1127, :1206-1210, :1371), outputs as fresh tensors, inputs never mutated.  The host path (checks,
allocations, autograd, launches) is native code, csrc/torch_op.cpp; this module gives it its Python names.

Differences, on purpose: gradients of factors that are broadcast over batch and/or heads are summed
over the broadcast dimensions (the reference indexes them with the un-expanded strides, :1227-1231);
a query row that sees no key yields 0 / -inf instead of NaN.
"""
from __future__ import annotations

import torch

from . import _lib

__all__ = ["FlashBiasFunc", "flash_bias_func", "flash_bias_forward", "flash_bias_backward",
           "FlashBiasAlibiFunc", "flash_bias_alibi_func", "check_device_status"]

_DT = {torch.float16: _lib.FB_DTYPE_F16, torch.bfloat16: _lib.FB_DTYPE_BF16, torch.float32: _lib.FB_DTYPE_F32}


def _strides_bhs(t: torch.Tensor):
    """(batch, head, row) element strides of a (B, S, H, C) tensor (a tuple: ctypes converts it on assignment)."""
    sb, ss, sh, _ = t.stride()
    return (sb, sh, ss)


def _factor_strides(t: torch.Tensor):
    """As above with 0 for broadcast (size-1) batch/head dims."""
    sb, ss, sh, _ = t.stride()
    return (0 if t.shape[0] == 1 else sb, 0 if t.shape[2] == 1 else sh, ss)


def _op():
    """The native operators (csrc/torch_op.cpp); raises if the package has not been built."""
    global _torch_op
    if _torch_op is None:
        _lib.load()  # the C ABI library they call: its absence has its own message
        from . import _torch_op as mod
        _torch_op = mod
    return _torch_op


_torch_op = None


def _status_word() -> torch.Tensor:
    """One int32 in pinned (device-visible) host memory: kernels store a device-side error code there, the host
    reads it without synchronising anything."""
    return _op().status_word()


def check_device_status() -> None:
    """Raise if a kernel of an earlier call reported a device-side error (a bounded wait that expired, a factor
    that overflowed the 16-bit type); the results of that call are invalid.  Called at the start of every
    forward and backward; callers can also call it after a synchronisation point of their own."""
    _op().check_device_status()


def _fill_common(p: _lib.FbParams, q, k, v, q_bias, k_bias, mask, causal, softmax_scale, flags, alibi_slopes=None):
    """The inputs of a problem in the C ABI's parameter block, for callers that bind the ABI themselves."""
    batch, seqlen_q, nheads, d = q.shape
    _, seqlen_k, _, _ = k.shape
    p.B, p.H, p.Sq, p.Sk, p.D = batch, nheads, seqlen_q, seqlen_k, d
    p.R = q_bias.shape[-1] if q_bias is not None else 0
    p.dtype = _DT[q.dtype]
    p.causal = 1 if causal else 0
    p.flags = flags
    p.softmax_scale = softmax_scale
    p.status = _status_word().data_ptr()
    if alibi_slopes is not None:
        p.alibi_slopes = alibi_slopes.data_ptr()
    p.q, p.k, p.v = q.data_ptr(), k.data_ptr(), v.data_ptr()
    p.q_stride, p.k_stride, p.v_stride = _strides_bhs(q), _strides_bhs(k), _strides_bhs(v)
    if q_bias is not None:
        p.q_bias, p.k_bias = q_bias.data_ptr(), k_bias.data_ptr()
        p.q_bias_stride, p.k_bias_stride = _factor_strides(q_bias), _factor_strides(k_bias)
    if mask is not None:
        p.mask = mask.data_ptr()
        p.mask_dtype = _DT[mask.dtype]
        # (1, seqlen_k) is tested first, as in the reference (:1120-1123)
        p.mask_kind = _lib.FB_MASK_VECTOR if mask.shape[2] == 1 else _lib.FB_MASK_MATRIX
        p.mask_stride = (0 if mask.shape[0] == 1 else mask.stride(0),
                         0 if mask.shape[1] == 1 else mask.stride(1),
                         0 if mask.shape[2] == 1 else mask.stride(2))
        # a mask with fewer batch entries than q is read periodically (entry b % n): Swin's shift mask
        p.mask_batch_period = mask.shape[0] if 1 < mask.shape[0] < batch else 0


def flash_bias_forward(q, k, v, q_bias=None, k_bias=None, mask=None, causal=False, softmax_scale=None, flags=0,
                       alibi_slopes=None):
    """Forward launch (the role of ``_flash_attn_forward``, flash_bias_triton.py:1100-1194).

    Returns (o, lse, softmax_scale); lse is fp32 of shape (B, H, ceil(Sq/128)*128).
    """
    return _op().forward(q, k, v, q_bias, k_bias, mask, causal, softmax_scale, flags, alibi_slopes)


def flash_bias_backward(do, q, k, v, o, q_bias, k_bias, lse, mask=None, causal=False, softmax_scale=None, flags=0,
                        alibi_slopes=None):
    """Backward launches (the role of ``_flash_attn_backward``, flash_bias_triton.py:1197-1342).

    Returns (dq, dk, dv, dq_bias, dk_bias); factor gradients have the shape of the factors.
    """
    return _op().backward(do, q, k, v, o, q_bias, k_bias, lse, mask, causal, softmax_scale, flags, alibi_slopes)


def _unit_rows(*ts):
    return [t if t is None or t.stride(-1) == 1 else t.contiguous() for t in ts]


class FlashBiasFunc(torch.autograd.Function):
    """The differentiable operator of ``flash_bias_func``.

    ``apply`` of this class is ``flash_bias_func``, the native node (csrc/torch_op.cpp).  ``forward`` and ``backward``
    are the same operator as static methods, for code that derives from the class or calls them with a context of its
    own.
    """

    @staticmethod
    def forward(ctx, q, k, v, q_bias=None, k_bias=None, mask=None, causal=False, softmax_scale=None):
        q, k, v, q_bias, k_bias = _unit_rows(q, k, v, q_bias, k_bias)
        ctx.factor_shapes = [None if t is None else t.shape for t in (q_bias, k_bias)]
        q_bias, k_bias = _op().narrow_expanded(q_bias), _op().narrow_expanded(k_bias)
        o, lse, ctx.softmax_scale = flash_bias_forward(q, k, v, q_bias, k_bias, mask, causal, softmax_scale)
        ctx.save_for_backward(q, k, v, o, q_bias, k_bias, lse, mask)
        ctx.causal = causal
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, q_bias, k_bias, lse, mask = ctx.saved_tensors
        assert not any(ctx.needs_input_grad[5:6]), "FlashBias does not support mask gradient yet"
        with torch.no_grad():
            dq, dk, dv, dq_bias, dk_bias = flash_bias_backward(do, q, k, v, o, q_bias, k_bias, lse, mask, ctx.causal,
                                                               ctx.softmax_scale)
            dq_bias, dk_bias = (g if g is None else _op().widen_grad(g, s)
                                for g, s in zip((dq_bias, dk_bias), ctx.factor_shapes))
        return dq, dk, dv, dq_bias, dk_bias, None, None, None

    @classmethod
    def apply(cls, *args, **kwargs):
        return flash_bias_func(*args, **kwargs) if cls is FlashBiasFunc else super().apply(*args, **kwargs)


def flash_bias_func(q, k, v, q_bias=None, k_bias=None, mask=None, causal=False, softmax_scale=None):
    """
    q: (batch_size, seqlen_q, nheads, headdim)
    k, v: (batch_size, seqlen_k, nheads, headdim)
    q_bias: (batch_size | 1, seqlen_q, nheads | 1, rankdim)
    k_bias: (batch_size | 1, seqlen_k, nheads | 1, rankdim)
    mask: optional, (batch | 1, nheads | 1, 1 | seqlen_q, seqlen_k), added to the logits.
    softmax_scale: multiplies q.k only; defaults to 1 / sqrt(headdim).
    """
    return (_torch_op or _op()).flash_bias(q, k, v, q_bias, k_bias, mask, causal, softmax_scale)


class FlashBiasAlibiFunc(torch.autograd.Function):
    """Attention with the ALiBi bias ``slopes[h] * (j - i)`` generated inside the kernels.

    The reference's language-model call site builds this bias as rank-2 factors from the positions and the
    per-head slopes (1_Language_Model/attention_with_alibi_bias.py:47-52) and feeds them to
    ``flash_bias_func``; here the slopes go in directly, the positions never exist as tensors and are never
    rounded to 16 bits.  ``slopes`` is an fp32 tensor of ``nheads`` values, a constant (the reference
    registers it as a buffer): it gets no gradient.  ``apply``, ``forward`` and ``backward``: as in ``FlashBiasFunc``.
    """

    @staticmethod
    def forward(ctx, q, k, v, slopes, causal=True, softmax_scale=None):
        q, k, v = _unit_rows(q, k, v)
        slopes = slopes.detach().to(device=q.device, dtype=torch.float32).reshape(-1).contiguous()
        assert slopes.numel() == q.shape[2], "one slope per head"
        o, lse, ctx.softmax_scale = flash_bias_forward(q, k, v, causal=causal, softmax_scale=softmax_scale,
                                                       alibi_slopes=slopes)
        ctx.save_for_backward(q, k, v, o, lse, slopes)
        ctx.causal = causal
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse, slopes = ctx.saved_tensors
        with torch.no_grad():
            dq, dk, dv, _, _ = flash_bias_backward(do, q, k, v, o, None, None, lse, None, ctx.causal, ctx.softmax_scale,
                                                   alibi_slopes=slopes)
        return dq, dk, dv, None, None, None

    @classmethod
    def apply(cls, *args, **kwargs):
        return flash_bias_alibi_func(*args, **kwargs) if cls is FlashBiasAlibiFunc else super().apply(*args, **kwargs)


def flash_bias_alibi_func(q, k, v, slopes, causal=True, softmax_scale=None):
    """The operator of ``FlashBiasAlibiFunc``."""
    return (_torch_op or _op()).flash_bias_alibi(q, k, v, slopes, causal, softmax_scale)
