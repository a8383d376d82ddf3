"""The single-query forward: one row per (batch, head) against the CPU checker, at the edges of its head groups, key
splits and rounds."""
import math

import pytest
import torch

from flashbias_b200 import check_device_status, flash_bias_alibi_func
from flashbias_b200.flash_bias import flash_bias_forward
from oracle import flashbias_oracle as orc
from tests.helpers import check_close, kernels_taken

pytestmark = pytest.mark.gpu

# (B, H, Sk, D, R, batch broadcast, mask, causal, dtype)
CASES = [
    (1, 1, 1, 32, 2, True, None, False, torch.bfloat16),         # one key
    (3, 50, 700, 32, 2, True, None, False, torch.bfloat16),      # one head group with idle lanes
    (2, 16, 2049, 32, 0, True, None, False, torch.float16),      # several keys side by side, splits with a remainder
    (1, 50, 5001, 64, 5, False, None, False, torch.float16),     # two head groups, many splits
    (2, 50, 300, 128, 20, True, None, False, torch.bfloat16),    # four head groups, two bias columns per lane
    (2, 3, 130, 24, 96, True, None, False, torch.bfloat16),      # rank that does not fit the lane group (tiled kernel)
    (2, 3, 130, 24, 15, True, None, False, torch.bfloat16),      # rows shorter than the lane group, four columns per lane
    (4, 2, 257, 8, 1, True, "vector", False, torch.bfloat16),    # one lane per head, key-padding mask
    (4, 6, 100, 16, 3, False, "matrix", False, torch.float16),   # periodic 16-bit mask
    (2, 4, 65, 32, 2, True, None, True, torch.bfloat16),         # causal, top-left aligned: the first key only
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "B%dH%dSk%dD%dR%d%s%s" % (*c[:5], "c" if c[7] else "", c[6] or ""))
def test_single_query_forward(case):
    B, H, Sk, D, R, bcast, mkind, causal, dtype = case
    g = torch.Generator().manual_seed(Sk + D)
    q = torch.randn(B, 1, H, D, generator=g).to(dtype)
    k, v = (torch.randn(B, Sk, H, D, generator=g).to(dtype) for _ in range(2))
    qb = kb = mask = None
    if R:
        qb, kb = ((torch.randn(1 if bcast else B, S, H, R, generator=g) * 0.5).to(dtype) for S in (1, Sk))
    if mkind:
        mask = torch.randn(B // 2 if mkind == "matrix" else B, 1, 1, Sk, generator=g)
        mask[..., Sk // 2:] = float("-inf") if mkind == "vector" else -50.0
        mask = mask.to(dtype if mkind == "matrix" else torch.float32)
    dev = [t.cuda() if t is not None else None for t in (q, k, v, qb, kb, mask)]
    assert kernels_taken(*dev, causal)[0] == ("fwd_tiled" if R == 96 else "fwd_one_query")
    o, lse, _ = flash_bias_forward(*dev, causal, None)
    torch.cuda.synchronize()
    check_device_status()
    f = [t.float() if t is not None else None for t in (q, k, v, qb, kb)]
    m = None if mask is None else mask.float().repeat(B // mask.shape[0], 1, 1, 1)
    o_ref, lse_ref = orc.attention_forward(*f, m, causal, 1.0 / math.sqrt(D))
    check_close("decode/B%dH%dSk%dD%dR%d" % case[:5], o, o_ref, dtype)
    assert (lse[:, :, :1].float().cpu() - lse_ref).abs().max().item() < 2e-2


def test_single_query_permuted_cache_and_slopes():
    """A (B, H, S, D) cache passed as a permuted view, and the slope producer."""
    B, H, Sk, D = 2, 6, 321, 64
    g = torch.Generator().manual_seed(9)
    q = torch.randn(B, 1, H, D, generator=g).half()
    k, v = (torch.randn(B, H, Sk, D, generator=g).half() for _ in range(2))
    slopes = torch.tensor([0.01 * (h + 1) for h in range(H)])
    o = flash_bias_alibi_func(q.cuda(), k.cuda().permute(0, 2, 1, 3), v.cuda().permute(0, 2, 1, 3), slopes.cuda(), False)
    j = torch.arange(Sk).double()
    qb = torch.stack([torch.zeros(1, H), torch.ones(1, H)], dim=-1)[None].double()
    kb = torch.stack([torch.ones(Sk, H).double(), slopes.double()[None] * j[:, None]], dim=-1)[None]
    o_ref, _ = orc.attention_forward(q, k.permute(0, 2, 1, 3), v.permute(0, 2, 1, 3), qb, kb, None, False, None,
                                     dtype=torch.float64)
    check_close("decode/permuted_slopes", o, o_ref, torch.float16)


def test_single_query_without_a_visible_key():
    q, k = torch.randn(2, 1, 2, 32).half().cuda(), torch.randn(2, 400, 2, 32).half().cuda()
    mask = torch.full((2, 1, 1, 400), float("-inf"), device="cuda")
    o, lse, _ = flash_bias_forward(q, k, k, None, None, mask)
    assert (o == 0).all() and (lse[..., 0] == float("-inf")).all()


@pytest.mark.parametrize("level", [-1e37, -8e37, -2e38])
@pytest.mark.parametrize("Sk", [3, 400])
def test_single_query_under_a_large_finite_mask(level, Sk):
    """Every key carries the same finite mask, however large: the probabilities are those of the unmasked row."""
    g = torch.Generator().manual_seed(11)
    q, k, v = (torch.randn(2, S, 2, 32, generator=g).half().cuda() for S in (1, Sk, Sk))
    o, lse, _ = flash_bias_forward(q, k, v, None, None, torch.full((2, 1, 1, Sk), level, device="cuda"))
    # next to such a mask every q.k vanishes (an fp32 ulp is 2^100 or more): the mean of the values
    want = v.float().mean(1, keepdim=True)
    assert (o.float() - want).abs().max().item() <= 2.0 ** -10 * want.abs().max().item()  # one rounding to fp16, fp32 sums
    assert ((lse[..., 0] - level) / level).abs().max().item() <= 2.0 ** -21  # two products by log2 e and ln 2, one sum
