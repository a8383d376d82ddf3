"""The two-stream forward kernel (head_dim 65 to 128) at odd and even numbers of key tiles, the edges of its tiles, ranks and
scale kinds, against the CPU checker; and repeated, since a race between its streams would show as different bits."""
import math

import pytest
import torch

from flashbias_b200 import check_device_status, flash_bias_alibi_func
from flashbias_b200.flash_bias import flash_bias_forward
from oracle import flashbias_oracle as orc
from tests.helpers import check_close, kernels_taken

pytestmark = pytest.mark.gpu
BF, HF = torch.bfloat16, torch.float16

# (B, H, Sq, Sk, D, R, causal, scale, dtype); R < 0: slopes
CASES = [
    (1, 2, 2, 1, 128, 0, False, None, BF),        # one key: the second stream has no tile
    (1, 2, 128, 128, 72, 2, False, None, HF),     # exactly one tile
    (1, 2, 129, 129, 128, 16, False, 0.125, BF),  # one past a tile, power-of-two scale (bf16: no split), full packed rank
    (2, 2, 200, 385, 128, 17, False, None, HF),   # four key tiles, packed rank 32
    (1, 2, 300, 300, 96, 32, True, None, BF),     # causal, 1 to 3 key tiles per item
    (1, 2, 450, 260, 128, 3, True, None, HF),     # causal, Sq > Sk
    (1, 2, 100, 700, 80, 0, True, None, BF),      # causal, Sq < Sk
    (3, 60, 257, 257, 128, 2, True, None, BF),    # more items than SMs
    (1, 4, 640, 640, 128, -1, True, None, HF),    # slopes
    (1, 4, 333, 641, 104, -1, False, None, BF),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "B%dH%dSq%dSk%dD%dR%d%s" % (*c[:6], "c" if c[6] else ""))
def test_edges(case):
    B, H, Sq, Sk, D, R, causal, scale, dtype = case
    scale = scale or 1.0 / math.sqrt(D)
    g = torch.Generator().manual_seed(Sq * 5 + Sk + D)
    q = torch.randn(B, Sq, H, D, generator=g).to(dtype)
    k, v = (torch.randn(B, Sk, H, D, generator=g).to(dtype) for _ in range(2))
    qb = kb = None
    if R > 0:
        qb, kb = ((torch.randn(1, S, H, R, generator=g) * 0.5).to(dtype) for S in (Sq, Sk))
    dev = [t.cuda() if t is not None else None for t in (q, k, v, qb, kb)]
    assert kernels_taken(*dev, causal=causal, slopes=torch.ones(H, device="cuda") if R < 0 else None)[0] == "fwd_two_stream"
    f = [t.float() if t is not None else None for t in (q, k, v, qb, kb)]
    if R < 0:
        m = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)])
        run = lambda: (flash_bias_alibi_func(*dev[:3], m.cuda(), causal, scale), None)
        m, i, j = m.double(), torch.arange(Sq).double(), torch.arange(Sk).double()
        f[3] = torch.stack([-(m[None] * i[:, None]), torch.ones(Sq, H).double()], dim=-1)[None]
        f[4] = torch.stack([torch.ones(Sk, H).double(), m[None] * j[:, None]], dim=-1)[None]
    else:
        run = lambda: flash_bias_forward(*dev, None, causal, scale)[:2]
    o, lse = run()
    torch.cuda.synchronize()
    check_device_status()
    o_ref, lse_ref = orc.attention_forward(*f, None, causal, scale, dtype=torch.float64)
    check_close("fwd_streams/Sq%dSk%dD%dR%d" % (Sq, Sk, D, R), o, o_ref, dtype)
    if lse is not None:  # fp32 sums of 16-bit products: 2^-22 of logits up to about 30
        assert (lse[..., :Sq].cpu().double() - lse_ref.double().reshape(B, H, -1)[..., :Sq]).abs().max() < 2e-5
    for _ in range(20):
        assert torch.equal(run()[0], o)


@pytest.mark.parametrize("tiles", [(2,), (3,), (3, 4), (2, 6), (5, 6)], ids=str)
def test_rescale_behind_tiles_without_one(tiles):
    """One key of each named tile raises the running maximum of every row by 2^20 or more, behind tiles that leave it alone: the
    accumulator is rescaled while the products of the tiles before may still be on their way into it."""
    B, H, Sq, Sk, D = 2, 40, 256, 7 * 128, 128  # more items than SMs
    g = torch.Generator().manual_seed(sum(tiles))
    q, k, v = (torch.randn(B, S, H, D, generator=g).to(BF) for S in (Sq, Sk, Sk))
    q[..., 0], k[..., 0] = 4.0, 0.0
    for n, t in enumerate(tiles):
        k[:, 128 * t + 77, :, 0] = 60.0 * (n + 1)  # a logit of 21 (n + 1); the others are N(0, 1)
    scale = 1.0 / math.sqrt(D)
    dev = [t.cuda() for t in (q, k, v)]
    run = lambda: flash_bias_forward(*dev, None, None, None, False, scale)[0]
    o = run()
    torch.cuda.synchronize()
    check_device_status()
    o_ref, _ = orc.attention_forward(q[:1, :, :8], k[:1, :, :8], v[:1, :, :8], None, None, None, False, scale, dtype=torch.float64)
    check_close("fwd_streams/rescale%s" % (tiles,), o[:1, :, :8], o_ref, BF)
    for _ in range(20):
        assert torch.equal(run(), o)


@pytest.mark.parametrize("D", [32, 64])
def test_causal_visits_keys_in_ascending_order_with_factors(D):
    """The last query sees every key with and without causal masking: the same tiles in the same order give the same bits.  (In
    another order P is rounded against another maximum; o then moves within its rounding, and an ALiBi dq_bias by 40 %.)"""
    B, H, S = 1, 8, 900
    g = torch.Generator().manual_seed(D)
    q, k, v = (torch.randn(B, S, H, D, generator=g).to(BF).cuda() for _ in range(3))
    m, i = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)]), torch.arange(S).float()
    one = torch.ones(S, H)
    qb = torch.stack([-(m[None] * i[:, None]), one], dim=-1)[None].to(BF).cuda()
    kb = torch.stack([one, m[None] * i[:, None]], dim=-1)[None].to(BF).cuda()
    run = lambda causal: flash_bias_forward(q, k, v, qb, kb, None, causal, 1.0 / math.sqrt(D))[0]
    assert torch.equal(run(True)[:, -1], run(False)[:, -1])
