"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one call pattern of a public entry point at one size.  The families follow the call sites the operator was
made for: causal language models with ALiBi (training, prompt processing, token generation), windowed vision
attention with a relative-position bias (training, and inference with the shifted-window mask behind the fp32 glue
kernel), solvers on point clouds with a distance bias, and structure models with a low-rank pair bias, plus the
operator's own benchmark shape.  ``listed()`` has one or two sizes of each family, ``draw()`` any size of its range.

Values: q, k, v and dO are N(0, 1); the factors are those of the family (positions times slopes, squared distances,
smooth position features, or i.i.d. values with the spread that a truncated SVD of a unit-variance bias has).
"""
import math

import torch

from flashbias_b200 import flash_bias_alibi_func, flash_bias_func
from flashbias_b200.layout import prepare_bhsd

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, family, B, H, Sq, Sk, D, R, dtype, train, **more):
    case = dict(family=family, B=B, H=H, Sq=Sq, Sk=Sk, D=D, R=R, dtype=dtype, train=train, **more)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the operator's benchmark shape (2 x 4 heads, head_dim 32, rank 8) at its shortest sequence: a small layer,
        # where the call itself and its launches are what a user waits for
        _case("generic_256_train", "generic", 2, 4, 256, 256, 32, 8, "fp16", True),
        # the same shape at 1024 tokens
        _case("generic_1k_train", "generic", 2, 4, 1024, 1024, 32, 8, "fp16", True),
        # a training step of a 50-head causal language model with ALiBi as rank-2 factors, 8192 tokens
        _case("alibi_8k_train", "alibi", 1, 50, 8192, 8192, 32, 2, "bf16", True),
        # the same bias from the per-head slopes, at the head_dim 128 of most present-day language models
        _case("slopes_d128_2k_train", "slopes", 2, 16, 2048, 2048, 128, 0, "bf16", True),
        # prompt processing (forward only) at head_dim 128, a prompt that fills no whole number of tiles
        _case("alibi_prefill_d128", "alibi", 1, 32, 4001, 4001, 128, 2, "fp16", False),
        # token generation: one new query per sequence against a key/value cache of odd length
        _case("alibi_decode", "decode", 16, 50, 1, 5001, 32, 2, "bf16", False),
        # windowed attention (16 x 16 tokens), rank-16 relative-position bias shared by all windows, training
        _case("windows_train", "windows", 4096, 24, 256, 256, 32, 16, "bf16", True),
        # inference of a shifted-window block: fp32 (B, H, S, D) activations through the glue kernel (cast, cosine
        # normalisation, logit scale), then the operator with the shift mask of 16 windows per image
        _case("windows_shift_infer", "shift", 1024, 8, 256, 256, 32, 16, "fp16", False, period=16),
        # a solver layer on a 32768-point cloud, squared-distance bias shared by the heads, training
        _case("points_32k_train", "points", 2, 8, 32768, 32768, 64, 5, "bf16", True),
        # pair-biased attention over 1536 tokens, rank 32 from an SVD per head, training
        _case("pair_1536_train", "pair", 1, 16, 1536, 1536, 32, 32, "bf16", True),
        # the same kind of layer at the head_dim 24 of a single representation, ragged token count
        _case("pair_d24_train", "pair", 1, 16, 743, 743, 24, 8, "bf16", True),
        # triangle attention inference: every row of the pair representation is a batch entry, rank-96 factors from a
        # network, shared by the batch, scale already in q
        _case("triangle_r96_infer", "triangle", 384, 4, 384, 384, 32, 96, "fp16", False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["generic", "alibi", "slopes", "prefill", "decode", "windows", "shift", "points", "pair",
                         "pair_odd", "triangle"])
    dtype = rng.choice(["bf16", "fp16"])
    if family == "generic":
        S = _log_int(rng, 128, 4096)
        return _case(None, "generic", rng.choice([1, 2, 3]), rng.choice([4, 6, 8]), S, S, rng.choice([32, 64]),
                     rng.randint(2, 8), dtype, True)
    if family == "alibi":
        S = _log_int(rng, 256, 8192)
        return _case(None, "alibi", 1, rng.choice([12, 25, 32, 50]), S, S, rng.choice([32, 64]), 2, "bf16", True)
    if family == "slopes":
        S = _log_int(rng, 256, 2048)
        return _case(None, "slopes", rng.choice([1, 2]), rng.choice([8, 12, 16]), S, S, rng.choice([32, 64, 128]), 0,
                     "bf16", True)
    if family == "prefill":
        S = _log_int(rng, 256, 8192)
        return _case(None, "alibi", 1, rng.choice([16, 25, 32]), S, S, rng.choice([32, 64, 128]), 2, dtype, False)
    if family == "decode":
        return _case(None, "decode", _log_int(rng, 1, 32), rng.choice([16, 25, 32, 50]), 1, _log_int(rng, 256, 8192),
                     rng.choice([32, 64, 128]), 2, dtype, False)
    if family == "windows":
        S = rng.choice([7, 8, 12, 14, 16, 24]) ** 2
        return _case(None, "windows", _log_int(rng, 64, 1024), rng.choice([3, 6, 12, 24]), S, S, 32, rng.randint(4, 16),
                     "bf16", True)
    if family == "shift":
        S = rng.choice([8, 12, 14, 16, 24]) ** 2
        period = rng.choice([4, 9, 16])
        return _case(None, "shift", period * _log_int(rng, 4, 64), rng.choice([4, 8, 16]), S, S, 32, rng.randint(4, 16),
                     "fp16", False, period=period)
    if family == "points":
        S = _log_int(rng, 1000, 32768)
        return _case(None, "points", rng.choice([1, 2]), rng.choice([4, 8]), S, S, rng.choice([32, 64]), 5, "bf16", True)
    if family == "pair":
        S = _log_int(rng, 128, 2048)
        return _case(None, "pair", 1, 16, S, S, 32, rng.choice([8, 16, 32]), "bf16", True)
    if family == "pair_odd":
        S = _log_int(rng, 128, 1024)
        return _case(None, "pair", 1, rng.choice([8, 16]), S, S, rng.choice([16, 24, 48]), rng.randint(4, 16), "bf16", True)
    S = _log_int(rng, 128, 640)
    return _case(None, "triangle", rng.choice([64, S]), 4, S, S, 32, 96, "fp16", False)


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _slopes(H, device):
    return torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)], dtype=torch.float32, device=device)


def _alibi_factors(H, Sq, Sk, device):
    """slope * (j - i) as rank-2 factors; the queries are the last Sq of the Sk positions."""
    m = _slopes(H, device)
    i = torch.arange(Sk - Sq, Sk, dtype=torch.float32, device=device)
    j = torch.arange(Sk, dtype=torch.float32, device=device)
    qb = torch.stack([-(m[None, :] * i[:, None]), torch.ones(Sq, H, device=device)], dim=-1)
    kb = torch.stack([torch.ones(Sk, H, device=device), m[None, :] * j[:, None]], dim=-1)
    return qb.unsqueeze(0), kb.unsqueeze(0)


def _window_factors(H, S, R, g, device):
    """Smooth features of the relative position: sums of cos(w . (y_i - y_j)), one pair of columns per frequency."""
    w = math.isqrt(S)
    ys, xs = torch.meshgrid(torch.arange(w, device=device), torch.arange(w, device=device), indexing="ij")
    pos = torch.stack([ys.flatten(), xs.flatten()], dim=-1).float() / w
    freq = torch.randn(2, H * ((R + 1) // 2), generator=g, device=device) * 3.0
    ph = (pos @ freq).reshape(S, H, (R + 1) // 2)
    f = torch.cat([torch.cos(ph), torch.sin(ph)], dim=-1)[..., :R] * (2.0 / math.sqrt(R))
    return f.unsqueeze(0), f.unsqueeze(0)


def _distance_factors(B, S, g, device, alpha=4.0):
    """-alpha |x_i - x_j|^2 for points uniform in the unit cube, exact rank 5, shared by the heads."""
    x = torch.rand(B, S, 3, generator=g, device=device)
    n2 = (x * x).sum(-1, keepdim=True)
    one = torch.ones_like(n2)
    qb = torch.cat([-alpha * n2, 2 * alpha * x, one], dim=-1).unsqueeze(2)
    kb = torch.cat([one, x, -alpha * n2], dim=-1).unsqueeze(2)
    return qb, kb


def _shift_mask(period, S, device):
    """(period, 1, S, S) fp32: -100 between tokens of different image regions in the windows of the last row and
    column of the window grid, 0 elsewhere."""
    w, grid = math.isqrt(S), math.isqrt(period)
    ys, xs = torch.meshgrid(torch.arange(w, device=device), torch.arange(w, device=device), indexing="ij")
    far = w - w // 2
    mask = torch.zeros(period, 1, S, S, device=device)
    for n in range(period):
        wy, wx = n // grid, n % grid
        region = (2 * ((ys >= far) & (wy == grid - 1)) + ((xs >= far) & (wx == grid - 1))).flatten()
        mask[n, 0] = torch.where(region[:, None] == region[None, :], 0.0, -100.0)
    return mask


def prepare(case, seed):
    device = torch.device("cuda")
    g = torch.Generator(device=device).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    family, train = case["family"], case["train"]
    B, H, Sq, Sk, D, R = (case[n] for n in ("B", "H", "Sq", "Sk", "D", "R"))

    def randn(*shape, dt=dtype):
        return torch.randn(shape, generator=g, device=device, dtype=dt)

    state = {"family": family, "train": train, "causal": family in ("alibi", "slopes"), "scale": 1.0 / math.sqrt(D)}
    if family == "shift":
        # the activations of the block as its projection leaves them: fp32, (B, H, S, D) slices of one buffer
        qkv = randn(3, B, H, Sq, D, dt=torch.float32)
        state["q"], state["k"], state["v"] = qkv[0], qkv[1], qkv[2]
        state["logit_scale"] = torch.rand(H, generator=g, device=device) * 5.0 + 5.0
        state["mask"] = _shift_mask(case["period"], Sq, device)
        state["scale"] = 1.0
    else:
        state["q"], state["k"], state["v"] = randn(B, Sq, H, D), randn(B, Sk, H, D), randn(B, Sk, H, D)
    if family == "triangle":
        state["q"] = state["q"] / math.sqrt(D)
        state["scale"] = 1.0
    if family == "slopes":
        state["slopes"] = _slopes(H, device)
    else:
        if family in ("alibi", "decode"):
            qb, kb = _alibi_factors(H, Sq, Sk, device)
        elif family in ("windows", "shift"):
            qb, kb = _window_factors(H, Sq, R, g, device)
        elif family == "points":
            qb, kb = _distance_factors(B, Sq, g, device)
        elif family == "pair":
            # U sqrt(s) of a truncated SVD of an N x N unit-variance bias: s ~ 2 sqrt(N), entries of U ~ 1 / sqrt(N)
            std = math.sqrt(2.0 / math.sqrt(Sq))
            qb, kb = randn(1, Sq, H, R) * std, randn(1, Sk, H, R) * std
        elif family == "triangle":
            qb, kb = torch.tanh(randn(1, Sq, H, R)) * 0.3, torch.tanh(randn(1, Sk, H, R)) * 0.3
        else:
            qb, kb = randn(B, Sq, H, R), randn(B, Sk, H, R)
        state["q_bias"], state["k_bias"] = qb.to(dtype).contiguous(), kb.to(dtype).contiguous()
    if train:
        state["do"] = randn(B, Sq, H, D)
        names = ["q", "k", "v"] + ([] if family == "slopes" else ["q_bias", "k_bias"])
        for n in names:
            state[n].requires_grad_(True)
        state["leaves"] = [state[n] for n in names]
    return state


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def run(state):
    s = state
    if s["train"]:
        if s["family"] == "slopes":
            o = flash_bias_alibi_func(s["q"], s["k"], s["v"], s["slopes"], s["causal"], s["scale"])
        else:
            o = flash_bias_func(s["q"], s["k"], s["v"], s["q_bias"], s["k_bias"], None, s["causal"], s["scale"])
        return (o,) + torch.autograd.grad(o, s["leaves"], s["do"])
    with torch.no_grad():
        if s["family"] == "shift":
            q = prepare_bhsd(s["q"], torch.float16, normalize=True, head_scale=s["logit_scale"])
            k = prepare_bhsd(s["k"], torch.float16, normalize=True)
            v = prepare_bhsd(s["v"], torch.float16)
            return flash_bias_func(q, k, v, s["q_bias"], s["k_bias"], s["mask"], False, s["scale"])
        return flash_bias_func(s["q"], s["k"], s["v"], s["q_bias"], s["k_bias"], None, s["causal"], s["scale"])


def work(case):
    """Bytes: every input read once, every output written once.  Flop: the attended (query, key) pairs times
    4 D + 2 R forward and 10 D + 6 R backward."""
    B, H, Sq, Sk, D, R = (case[n] for n in ("B", "H", "Sq", "Sk", "D", "R"))
    family = case["family"]
    causal = family in ("alibi", "slopes")
    pairs = B * H * (Sq * (Sq + 1) // 2 if causal else Sq * Sk)
    fB = B if family in ("generic", "points") else 1
    fH = 1 if family == "points" else H
    factors = 2 * fB * fH * (Sq + Sk) * R
    q, kv = 2 * B * H * Sq * D, 2 * 2 * B * H * Sk * D
    if family == "shift":
        nbytes = 2 * (q + kv) + factors + 4 * case["period"] * Sq * Sk + q
    elif case["train"]:
        nbytes = (q + kv + factors + q) + (q + q + kv + factors)
    else:
        nbytes = q + kv + factors + q
    flops = pairs * (4.0 * D + 2.0 * R)
    if case["train"]:
        flops += pairs * (10.0 * D + 6.0 * R)
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """16-bit results from products whose probabilities are rounded to the same 16 bits."""
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
