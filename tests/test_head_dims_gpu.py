"""Head dimensions that run in the next wider tile (zero-filled columns), and the head_dim-128 backward without factor
operands, at the edges of their tiles: forward, lse and gradients against the CPU checker."""
import math

import pytest
import torch

from flashbias_b200 import check_device_status, flash_bias_alibi_func, flash_bias_func
from oracle import flashbias_oracle as orc
from tests.helpers import check_close, kernels_taken

pytestmark = pytest.mark.gpu

# (B, H, Sq, Sk, D, R, causal, mode, dtype); mode: "plain", "mask" or "slopes"
CASES = [
    (2, 3, 130, 130, 8, 3, False, "plain", torch.bfloat16),       # narrowest row, ragged
    (1, 2, 257, 129, 16, 8, True, "plain", torch.float16),        # causal, Sq > Sk
    (1, 4, 200, 300, 24, 12, False, "mask", torch.bfloat16),      # cross attention with a mask
    (40, 8, 144, 144, 24, 8, False, "plain", torch.bfloat16),     # many short items: persistent form, clipped tile stores
    (1, 2, 140, 140, 40, 0, True, "slopes", torch.bfloat16),
    (1, 2, 333, 333, 48, 5, False, "plain", torch.float16),
    (1, 2, 64, 200, 56, 0, True, "plain", torch.bfloat16),        # causal, Sq < Sk: key tiles that no query sees
    (1, 2, 190, 190, 72, 0, True, "slopes", torch.bfloat16),      # head_dim 128 tile, one column block of 8
    (1, 2, 65, 3, 128, 0, False, "plain", torch.float16),         # three keys; one row past a 64-row tile
    (2, 2, 1, 130, 96, 0, False, "plain", torch.bfloat16),        # a single query
    (1, 3, 64, 128, 128, 0, True, "plain", torch.bfloat16),       # exactly one tile each
    (1, 2, 100, 300, 128, 0, True, "plain", torch.bfloat16),      # causal, Sq < Sk
    (2, 2, 450, 260, 128, 0, True, "slopes", torch.bfloat16),     # several tiles, causal, Sq > Sk
    (1, 2, 200, 333, 128, 0, False, "mask", torch.float16),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "B%dH%dSq%dSk%dD%dR%d%s_%s" % (*c[:6], "c" if c[6] else "", c[7]))
def test_head_dims(case):
    B, H, Sq, Sk, D, R, causal, mode, dtype = case
    g = torch.Generator().manual_seed(D * 1000 + Sq)
    q, do = (torch.randn(B, Sq, H, D, generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, Sk, H, D, generator=g).to(dtype) for _ in range(2))
    qb = kb = mask = None
    if R:
        qb, kb = ((torch.randn(1, S, H, R, generator=g) * 0.5).to(dtype) for S in (Sq, Sk))
    if mode == "mask":
        mask = torch.where(torch.rand(B, 1, Sq, Sk, generator=g) < 0.3, -100.0, torch.randn(B, 1, Sq, Sk, generator=g))
    leaves = [t.cuda().requires_grad_(True) for t in (q, k, v, qb, kb) if t is not None]
    f = [t.float() for t in (q, k, v)] + [t.float() if t is not None else None for t in (qb, kb)]
    slopes_dev = torch.ones(H, device="cuda") if mode == "slopes" else None
    dev = [t.detach() for t in leaves] + [None] * (5 - len(leaves))
    bwd = ("bwd_key_major" if D > 64 else "bwd_persistent" if B == 40 else "bwd_query_major" if mode == "mask" else "bwd_two_stream")
    assert kernels_taken(*dev, mask.cuda() if mask is not None else None, causal, 0, slopes_dev) == (
        "fwd_one_query" if Sq == 1 else "fwd_two_stream" if D > 64 and mode != "mask" else "fwd_tiled", bwd)
    if mode == "slopes":
        slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)])
        o = flash_bias_alibi_func(*leaves, slopes.cuda(), causal)
        m, i, j = slopes.double(), torch.arange(Sq).double(), torch.arange(Sk).double()
        f[3] = torch.stack([-(m[None] * i[:, None]), torch.ones(Sq, H).double()], dim=-1)[None]
        f[4] = torch.stack([torch.ones(Sk, H).double(), m[None] * j[:, None]], dim=-1)[None]
    else:
        o = flash_bias_func(*leaves, *([None, None] if not R else []), mask.cuda() if mask is not None else None, causal)
    grads = torch.autograd.grad(o, leaves, do.cuda())
    torch.cuda.synchronize()
    check_device_status()
    scale = 1.0 / math.sqrt(D)
    o_ref, lse_ref = orc.attention_forward(*f, mask, causal, scale, dtype=torch.float64)
    tag = "head_dim/D%dSq%dSk%d%s" % (D, Sq, Sk, mode)
    check_close(f"{tag}/o", o, o_ref, dtype)
    want = orc.attention_backward(do, *f[:3], o.detach().cpu(), lse_ref, f[3], f[4], mask, causal, scale, dtype=torch.float64)
    for name, got, ref in zip(("dq", "dk", "dv", "dq_bias", "dk_bias"), grads, want):
        check_close(f"{tag}/{name}", got, ref, dtype)
