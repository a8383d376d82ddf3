"""Mask tiles through the forward's TMA ring: element types, ragged and causal tiles, broadcast, periodic and per-head
masks, strided rows, and a mask whose rows TMA cannot address beside one that it can."""
import math

import pytest
import torch

from flashbias_b200 import check_device_status
from flashbias_b200.flash_bias import flash_bias_forward
from oracle import flashbias_oracle as orc
from tests.helpers import check_close

pytestmark = pytest.mark.gpu

# (B, H, Sq, Sk, D, R, causal, mask batch, mask heads, mask dtype, dtype)
CASES = [
    (40, 8, 256, 256, 32, 16, False, 4, 1, torch.float32, torch.float16),     # many items per CTA, periodic
    (40, 8, 144, 144, 32, 16, False, 40, 8, torch.float16, torch.float16),    # 16-bit, a mask of its own for every head
    (2, 3, 200, 328, 32, 0, False, 1, 3, torch.bfloat16, torch.bfloat16),     # ragged in both directions
    (1, 4, 130, 260, 64, 5, True, 1, 1, torch.float32, torch.bfloat16),       # causal, Sq < Sk: tiles beyond the diagonal
    (2, 2, 300, 516, 64, 40, False, 2, 1, torch.float32, torch.float16),      # packed rank 64
    (1, 2, 264, 400, 128, 20, False, 1, 2, torch.bfloat16, torch.bfloat16),   # head_dim 128
    (2, 2, 256, 384, 32, 70, False, 2, 2, torch.float32, torch.bfloat16),     # packed rank 128
    (2, 2, 196, 49, 32, 8, False, 2, 1, torch.float32, torch.bfloat16),       # rows of 196 bytes: not addressable by TMA
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "B%dH%dSq%dSk%dD%dR%d%s" % (*c[:6], "c" if c[6] else ""))
@pytest.mark.parametrize("padded_rows", [False, True])
def test_masked_forward(case, padded_rows):
    B, H, Sq, Sk, D, R, causal, mB, mH, mdtype, dtype = case
    g = torch.Generator().manual_seed(Sq + Sk + D)
    q = torch.randn(B, Sq, H, D, generator=g).to(dtype)
    k, v = (torch.randn(B, Sk, H, D, generator=g).to(dtype) for _ in range(2))
    qb = kb = None
    if R:
        qb, kb = ((torch.randn(1, S, H, R, generator=g) * 0.5).to(dtype) for S in (Sq, Sk))
    mask = torch.randn(mB, mH, Sq, Sk, generator=g)
    mask = torch.where(torch.rand(mB, mH, Sq, Sk, generator=g) < 0.2, torch.tensor(-100.0), mask).to(mdtype)
    mask[..., Sq // 2, 1:] = float("-inf")  # a row that sees one key
    mdev = torch.zeros(mB, mH, Sq, Sk + 24, dtype=mdtype, device="cuda")[..., :Sk] if padded_rows else torch.empty_like(mask, device="cuda")
    mdev.copy_(mask)
    dev = [t.cuda() if t is not None else None for t in (q, k, v, qb, kb)]
    o, lse, _ = flash_bias_forward(*dev, mdev, causal, None)
    torch.cuda.synchronize()
    check_device_status()
    f = [t.float() if t is not None else None for t in (q, k, v, qb, kb)]
    m = mask.float().repeat(B // mB, 1, 1, 1) if mB > 1 else mask.float()
    o_ref, lse_ref = orc.attention_forward(*f, m, causal, 1.0 / math.sqrt(D))
    check_close("mask_ring/B%dSq%dSk%dD%dR%d%s" % (B, Sq, Sk, D, R, "p" if padded_rows else ""), o, o_ref, dtype)
    assert (lse[:, :, :Sq].float().cpu() - lse_ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("mdtype", [torch.float32, torch.float16])
def test_repeated_masked_forward_is_bit_identical(mdtype):
    """Stages of the ring are reused as soon as they are released: a release ahead of the last read shows as rows that
    differ from run to run."""
    g = torch.Generator().manual_seed(6)
    q, k, v = (torch.randn(64, 256, 8, 32, generator=g).half().cuda() for _ in range(3))
    qb, kb = ((torch.randn(1, 256, 8, 16, generator=g) * 0.5).half().cuda() for _ in range(2))
    mask = torch.randn(4, 1, 256, 256, generator=g).to(mdtype).cuda()
    unaligned = torch.zeros(4, 1, 256, 257, dtype=mdtype, device="cuda")[..., :256].copy_(mask)  # read without the ring
    want, _, _ = flash_bias_forward(q, k, v, qb, kb, unaligned)
    for _ in range(50):
        got, _, _ = flash_bias_forward(q, k, v, qb, kb, mask)
        assert torch.equal(got, want)


# (head_dim, rank, softmax_scale, dtype): each number of mask stages (1 to 4), beside one and two CTAs per SM
RINGS = [
    (32, 0, None, torch.float16),     # 4 stages, two CTAs
    (32, 20, None, torch.bfloat16),   # 2 stages, two CTAs
    (32, 40, 0.25, torch.bfloat16),   # 1 stage, two CTAs
    (64, 0, None, torch.float16),     # 1 stage, two CTAs
    (32, 70, None, torch.bfloat16),   # 4 stages, one CTA
    (64, 70, 0.125, torch.bfloat16),  # 3 stages, one CTA
    (128, 0, None, torch.bfloat16),   # 4 stages, one CTA
    (128, 20, 0.25, torch.bfloat16),  # 2 stages, one CTA
    (128, 12, None, torch.float16),   # 1 stage, one CTA
]


@pytest.mark.parametrize("wide", [True, False], ids=["fp32", "16bit"])
@pytest.mark.parametrize("ring", RINGS, ids=lambda r: "D%dR%d" % r[:2])
def test_every_ring_depth_repeats_bit_identical(ring, wide):
    D, R, scale, dtype = ring
    mdtype = torch.float32 if wide else dtype
    g = torch.Generator().manual_seed(D + R)
    q, k, v = (torch.randn(48, 384, 8, D, generator=g).to(dtype).cuda() for _ in range(3))
    qb = kb = None
    if R:
        qb, kb = ((torch.randn(1, 384, 8, R, generator=g) * 0.3).to(dtype).cuda() for _ in range(2))
    mask = torch.randn(4, 1, 384, 384, generator=g).to(mdtype).cuda()
    unaligned = torch.zeros(4, 1, 384, 385, dtype=mdtype, device="cuda")[..., :384].copy_(mask)  # read without the ring
    want, _, _ = flash_bias_forward(q, k, v, qb, kb, unaligned, False, scale)
    for _ in range(30):
        got, _, _ = flash_bias_forward(q, k, v, qb, kb, mask, False, scale)
        assert torch.equal(got, want)
