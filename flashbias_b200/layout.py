"""Caller-side layout glue of the FlashBias call sites, fused into one pass.

The reference's call sites hold (B, H, S, D) tensors (often fp32) and run
``x.permute(0, 2, 1, 3).contiguous().half()`` -- Swin-V2 also ``F.normalize(q, dim=-1) * logit_scale`` -- on
each of q, k, v before every call (2_Vision_Transformer/swin_transformer_v2.py:194-199,
4_AlphaFold3/protenix/openfold_local/model/primitives.py:636-640).  ``prepare_bhsd`` does the cast, the
optional normalisation and the optional per-head scale in ONE kernel that reads the tensor where it lies
and writes a 16-bit tensor in the same (B, H, S, D) layout; the value returned is its (B, S, H, D) *view*,
which ``flash_bias_func`` takes as it is (the C ABI addresses batch, head and row through strides).
A 16-bit (B, H, S, D) tensor that needs neither normalisation nor scale needs no kernel at all:
``x.permute(0, 2, 1, 3)`` is already a valid argument.
"""
from __future__ import annotations

from typing import Optional

import torch

from .flash_bias import _op

__all__ = ["prepare_bhsd"]


def prepare_bhsd(x: torch.Tensor, dtype: torch.dtype = torch.float16, normalize: bool = False,
                 head_scale: Optional[torch.Tensor] = None, eps: float = 1e-12) -> torch.Tensor:
    """``x``: (B, H, S, D) CUDA tensor, any batch/head/row strides, rows contiguous, fp32/fp16/bf16.
    Returns the (B, S, H, D) view of a new ``dtype`` tensor holding ``normalize?(x) * head_scale[h]``."""
    return _op().prepare_bhsd(x, dtype, normalize, head_scale, eps)
