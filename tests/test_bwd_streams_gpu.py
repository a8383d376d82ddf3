"""The two-stream backward kernel at the edges of its tiles (64-query halves, 128-key tiles), ranks and scale kinds, against the
CPU oracle; and repeated, since a race between its two streams would show as a different gradient."""
import math

import pytest
import torch

from flashbias_b200 import check_device_status, flash_bias_alibi_func, flash_bias_func
from flashbias_b200.flash_bias import flash_bias_backward, flash_bias_forward
from oracle import flashbias_oracle as orc
from tests.helpers import check_close, kernels_taken

pytestmark = pytest.mark.gpu
BF, HF = torch.bfloat16, torch.float16

# (B, H, Sq, Sk, D, R, causal, scale, dtype, shared): R < 0: slopes; shared: factors without batch and head extent
CASES = [
    (1, 2, 1, 128, 32, 4, False, None, BF, False),       # one query, one key tile
    (1, 2, 64, 2, 32, 3, False, 0.25, BF, False),        # exactly one half; power-of-two scale; two keys (with one, dq and
                                                         # dk are zero and a relative bound says nothing)
    (2, 2, 65, 129, 32, 16, False, None, HF, True),      # one past a half and past a key tile, full packed rank
    (1, 3, 191, 127, 32, 17, False, None, BF, False),    # packed rank 32, second half ragged
    (1, 2, 128, 300, 32, 32, True, None, HF, False),     # causal, Sq < Sk, highest rank
    (1, 2, 450, 260, 32, 9, True, 0.5, BF, True),        # causal, Sq > Sk
    (1, 2, 700, 700, 32, -1, True, None, BF, False),
    (1, 2, 193, 400, 24, 0, False, None, HF, False),     # no factors, clipped columns
    (1, 2, 130, 130, 40, 8, True, None, BF, False),      # head_dim 64 tile
    (2, 1, 577, 321, 64, 1, False, None, BF, False),
    (1, 2, 256, 256, 64, 8, True, 0.1, HF, True),        # split scale at head_dim 64
    (1, 2, 63, 640, 64, 0, True, None, BF, False),
    (1, 2, 384, 384, 64, -1, True, None, HF, False),
]


def _inputs(case):
    B, H, Sq, Sk, D, R, _, _, dtype, shared = case
    g = torch.Generator().manual_seed(Sq * 7 + Sk + D)
    q, do = (torch.randn(B, Sq, H, D, generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, Sk, H, D, generator=g).to(dtype) for _ in range(2))
    qb = kb = None
    if R > 0:
        qb, kb = ((torch.randn(1, S, 1 if shared else H, R, generator=g) * 0.5).to(dtype) for S in (Sq, Sk))
    return q, k, v, qb, kb, do


@pytest.mark.parametrize("case", CASES, ids=lambda c: "B%dH%dSq%dSk%dD%dR%d%s" % (*c[:6], "c" if c[6] else ""))
def test_edges(case):
    B, H, Sq, Sk, D, R, causal, scale, dtype, _ = case
    scale = scale or 1.0 / math.sqrt(D)
    q, k, v, qb, kb, do = _inputs(case)
    leaves = [t.cuda().requires_grad_(True) for t in (q, k, v, qb, kb) if t is not None]
    slopes = torch.ones(H, device="cuda") if R < 0 else None
    assert kernels_taken(*(t.detach() for t in leaves), causal=causal, slopes=slopes)[1] == "bwd_two_stream"
    f = [t.float() if t is not None else None for t in (q, k, v, qb, kb)]
    if R < 0:
        m = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)])
        o = flash_bias_alibi_func(*leaves, m.cuda(), causal, scale)
        m, i, j = m.double(), torch.arange(Sq).double(), torch.arange(Sk).double()
        f[3] = torch.stack([-(m[None] * i[:, None]), torch.ones(Sq, H).double()], dim=-1)[None]
        f[4] = torch.stack([torch.ones(Sk, H).double(), m[None] * j[:, None]], dim=-1)[None]
    else:
        o = flash_bias_func(*leaves, *([None, None] if not R else []), None, causal, scale)
    grads = torch.autograd.grad(o, leaves, do.cuda())
    torch.cuda.synchronize()
    check_device_status()
    _, lse_ref = orc.attention_forward(*f, None, causal, scale, dtype=torch.float64)
    want = orc.attention_backward(do, *f[:3], o.detach().cpu(), lse_ref, f[3], f[4], None, causal, scale, dtype=torch.float64)
    for name, got, ref in zip(("dq", "dk", "dv", "dq_bias", "dk_bias"), grads, want):
        check_close("streams/Sq%dSk%dD%dR%d/%s" % (Sq, Sk, D, R, name), got, ref, dtype)


@pytest.mark.parametrize("D", [32, 64, 128])
def test_slopes_far_from_the_first_query(D):
    """The slopes' term counted from query 0 is a difference of two numbers as large as the position: at 65500 and slope 0.9 their
    fp32 rounding alone moves P by 1e-3 in the mean.  The last queries' dq, and dk and dv of the last keys, which no other query
    sees, against 64 bits."""
    S, H, n = 65500, 2, 96
    g = torch.Generator().manual_seed(D)
    q, k, v, do = (torch.randn(1, S, H, D, generator=g).to(HF) for _ in range(4))
    m = torch.tensor([0.9, 0.5])
    leaves = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    o = flash_bias_alibi_func(*leaves, m.cuda(), True)
    grads = torch.autograd.grad(o, leaves, do.cuda())
    torch.cuda.synchronize()
    check_device_status()
    i, j = torch.arange(S - n, S).double()[:, None], torch.arange(S).double()[None]
    bias = torch.where(j > i, -math.inf, m.double()[:, None, None] * (j - i))[None]
    last = [q[:, -n:], k, v]
    o_ref, lse_ref = orc.attention_forward(*last, None, None, bias, False, dtype=torch.float64)
    check_close("streams/far_D%d/o" % D, o[:, -n:], o_ref, HF)
    want = orc.attention_backward(do[:, -n:], *last, o[:, -n:].detach().cpu(), lse_ref, None, None, bias, False, dtype=torch.float64)
    for name, got, ref in zip(("dq", "dk", "dv"), grads, want):
        check_close("streams/far_D%d/%s" % (D, name), got[:, -n:], ref[:, -n:], HF)


# (both dS^T tiles; one dS^T tile; P^T in the place of S^T)
@pytest.mark.parametrize("case", [(2, 8, 1000, 1000, 32, 8, True, None, BF, False), (2, 8, 777, 777, 64, 5, False, 0.1, BF, False),
                                  (1, 16, 900, 900, 32, 30, False, None, BF, False)], ids=lambda c: "D%dR%d" % (c[4], c[5]))
def test_repeated_backward_is_bit_identical(case):
    """dk and dv bit for bit.  dq and the factor gradients, the readers of dS^T in shared memory and of the row-sum tables, are
    fp32 sums over the key tiles in no fixed order: at most 32 terms, each no more than 4 times the largest result, so 2^-17 of that
    ahead of the rounding, and a rounding that falls the other way.  Such a flip needs a sum within 2^-20 or so of its size from the
    middle of two 16-bit values, one in some thousand: 4e-5 in norm at bf16's 2^-8."""
    q, k, v, qb, kb, do = (t.cuda() for t in _inputs(case))
    assert kernels_taken(q, k, v, qb, kb, causal=case[6])[1] == "bwd_two_stream"
    o, lse, sc = flash_bias_forward(q, k, v, qb, kb, None, case[6], case[7])
    want = flash_bias_backward(do, q, k, v, o, qb, kb, lse, None, case[6], sc)
    for _ in range(60):
        got = flash_bias_backward(do, q, k, v, o, qb, kb, lse, None, case[6], sc)
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
        for a, b in zip((got[0], *got[3:]), (want[0], *want[3:])):
            d, b = (a.float() - b.float()).abs(), b.float()
            assert d.norm() <= 2e-4 * b.norm()
            assert (d <= torch.finfo(a.dtype).eps * torch.maximum(a.float().abs(), b.abs()) + 2.0 ** -17 * b.abs().max()).all()
    torch.cuda.synchronize()
    check_device_status()
