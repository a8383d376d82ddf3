"""The native host path of the operators: error behaviour inside autograd, strided masks in both directions, calls from
several threads at once, and the two ways to obtain delta in the C ABI."""
import math
import threading

import pytest
import torch

from flashbias_b200 import check_device_status, flash_bias_func
from oracle import flashbias_oracle as orc
from tests.helpers import check_close

pytestmark = pytest.mark.gpu


def _inputs(B, S, H, D, R, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    q, k, v, do = (torch.randn(B, S, H, D, generator=g).to(dtype) for _ in range(4))
    qb, kb = ((torch.randn(1, S, H, R, generator=g) * 0.5).to(dtype) for _ in range(2))
    return q, k, v, qb, kb, do


def test_mask_gradient_is_refused_in_backward():
    q, k, v, _, _, do = (t.cuda() for t in _inputs(1, 128, 2, 32, 4, torch.float16, 1))
    mask = torch.zeros(1, 1, 128, 128, device="cuda", requires_grad=True)
    o = flash_bias_func(q.requires_grad_(True), k, v, None, None, mask)
    with pytest.raises(AssertionError, match="mask gradient"):
        o.backward(do)
    (dq,) = torch.autograd.grad(flash_bias_func(q, k, v, None, None, mask), [q], do)  # the mask's gradient is not asked for
    assert torch.isfinite(dq).all()


def test_mask_without_batch_entries_is_refused():
    q, k, v, _, _, _ = (t.cuda() for t in _inputs(2, 32, 2, 32, 4, torch.float16, 1))
    with pytest.raises(AssertionError):
        flash_bias_func(q, k, v, None, None, torch.zeros(0, 1, 32, 32, device="cuda"))


@pytest.mark.parametrize("on_host", ["q", "k"])
def test_factors_in_host_memory_are_refused(on_host):
    q, k, v, qb, kb, _ = (t.cuda() for t in _inputs(1, 32, 2, 32, 4, torch.float16, 1))
    with pytest.raises(AssertionError):
        flash_bias_func(q, k, v, qb.cpu() if on_host == "q" else qb, kb.cpu() if on_host == "k" else kb)


def test_pinned_factors_are_read_in_place():
    q, k, v, qb, kb, _ = (t.cuda() for t in _inputs(1, 32, 2, 32, 4, torch.float16, 1))
    assert torch.equal(flash_bias_func(q, k, v, qb.cpu().pin_memory(), kb.cpu().pin_memory()), flash_bias_func(q, k, v, qb, kb))


@pytest.mark.parametrize("what", ["do_rows", "do_type", "o_rows", "k_heads", "factor_rows", "factors_on_host", "lse_type"])
def test_backward_refuses_what_its_kernels_would_misread(what):
    from flashbias_b200.flash_bias import flash_bias_backward, flash_bias_forward
    q, k, v, qb, kb, do = (t.cuda() for t in _inputs(2, 64, 2, 32, 4, torch.float16, 1))
    o, lse, _ = flash_bias_forward(q, k, v, qb, kb)
    args = dict(do=do, q=q, k=k, v=v, o=o, q_bias=qb, k_bias=kb, lse=lse)
    assert torch.isfinite(flash_bias_backward(**args)[0]).all()
    bad = {"do_rows": dict(do=do[:, :32]), "do_type": dict(do=do.float()), "o_rows": dict(o=o[:1]), "k_heads": dict(k=k[:, :, :1]),
           "factor_rows": dict(k_bias=kb[:, :32]), "factors_on_host": dict(q_bias=qb.cpu(), k_bias=kb.cpu()),
           "lse_type": dict(lse=lse.half())}[what]
    with pytest.raises(AssertionError):
        flash_bias_backward(**{**args, **bad})


@pytest.mark.parametrize("expanded", [False, True])
def test_a_derived_function_gives_the_operator_s_results(expanded):
    """Code may derive from FlashBiasFunc and call its forward and backward: the same values as the native node."""
    from flashbias_b200 import FlashBiasFunc
    seen = []

    class Logged(FlashBiasFunc):
        @staticmethod
        def forward(ctx, *args):
            seen.append("forward")
            return FlashBiasFunc.forward(ctx, *args)

        @staticmethod
        def backward(ctx, do):
            seen.append("backward")
            return FlashBiasFunc.backward(ctx, do)

    q, k, v, qb, kb, do = (t.cuda() for t in _inputs(2, 130, 2, 32, 4, torch.float16, 4))
    results = []
    for fn in (FlashBiasFunc, Logged):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v, qb, kb)]
        factors = [t.expand(2, -1, -1, -1) if expanded else t for t in leaves[3:]]
        o = fn.apply(*leaves[:3], *factors)
        results.append((o, *torch.autograd.grad(o, leaves, do)))
    assert seen == ["forward", "backward"]
    for a, b in zip(*results):  # fp32 sums over key tiles are not ordered: equal up to one rounding
        assert a.shape == b.shape and (a.float() - b.float()).abs().max() <= 2.0 ** -10 * b.float().abs().max()


def test_a_derived_function_takes_three_arguments():
    from flashbias_b200 import FlashBiasFunc
    q, k, v, _, _, do = (t.cuda() for t in _inputs(1, 64, 2, 32, 4, torch.float16, 4))
    o = type("Derived", (FlashBiasFunc,), {}).apply(q.requires_grad_(True), k, v)
    (dq,) = torch.autograd.grad(o, [q], do)
    (want,) = torch.autograd.grad(flash_bias_func(q, k, v), [q], do)
    assert (dq.float() - want.float()).abs().max() <= 2.0 ** -10 * want.float().abs().max()


def test_a_function_derived_from_the_slope_form():
    from flashbias_b200 import FlashBiasAlibiFunc
    q, k, v, _, _, do = (t.cuda() for t in _inputs(1, 130, 2, 32, 4, torch.float16, 4))
    slopes = torch.tensor([0.5, 0.25], device="cuda")
    results = []
    for fn in (FlashBiasAlibiFunc, type("Derived", (FlashBiasAlibiFunc,), {})):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        o = fn.apply(*leaves, slopes)
        results.append((o, *torch.autograd.grad(o, leaves, do)))
    for a, b in zip(*results):
        assert (a.float() - b.float()).abs().max() <= 2.0 ** -10 * b.float().abs().max()


def test_mask_with_strided_rows_is_read_right_in_both_directions():
    q, k, v, qb, kb, do = _inputs(2, 160, 2, 32, 4, torch.float16, 2)
    base = torch.randn(2, 1, 160, 320, generator=torch.Generator().manual_seed(3))
    dev = [t.cuda() for t in (q, k, v, qb, kb)]
    leaves = [t.requires_grad_(True) for t in dev]
    o = flash_bias_func(*leaves, base.cuda()[..., ::2])
    grads = torch.autograd.grad(o, leaves, do.cuda())
    f = [t.float() for t in (q, k, v, qb, kb)]
    o_ref, lse_ref = orc.attention_forward(*f, base[..., ::2])
    check_close("strided_mask/o", o, o_ref, torch.float16)
    g_ref = orc.attention_backward(do.float(), *f[:3], o.detach().float().cpu(), lse_ref, *f[3:], base[..., ::2])
    for name, got, want in zip(("dq", "dk", "dv", "dq_bias", "dk_bias"), grads, g_ref):
        check_close(f"strided_mask/{name}", got, want, torch.float16)


@pytest.mark.parametrize("own_stream", [False, True])
def test_threads_do_not_share_scratch(own_stream):
    """Forward + backward from four threads at once, on one stream and on a stream each: the results of each thread are
    those of a single-threaded call."""
    sets = [[t.cuda() for t in _inputs(2, 200 + 64 * i, 4, 32, 3 + i, torch.bfloat16, 10 + i)] for i in range(4)]

    def step(s):
        leaves = [t.detach().clone().requires_grad_(True) for t in s[:5]]
        o = flash_bias_func(*leaves)
        return (o,) + torch.autograd.grad(o, leaves, s[5])

    want = [step(s) for s in sets]
    torch.cuda.synchronize()
    got = [[] for _ in sets]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.current_stream()):
            for _ in range(20):
                got[i].append(step(sets[i]))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    check_device_status()
    for i, ref in enumerate(want):
        assert len(got[i]) == 20
        for res in got[i]:
            for a, b in zip(res, ref):  # fp32 sums over key tiles are not ordered: equal up to one rounding
                assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max()


@pytest.mark.parametrize("D,R,flags", [(32, 3, 0), (64, 8, 0), (40, 9, 1)])
def test_delta_taken_by_the_backward_equals_the_separate_pre_pass(D, R, flags):
    import ctypes as C

    from flashbias_b200 import _lib
    from flashbias_b200.flash_bias import _fill_common, _strides_bhs, flash_bias_forward
    q, k, v, qb, kb, do = (t.cuda() for t in _inputs(2, 130, 3, D, R, torch.bfloat16, 5))
    o, lse, sc = flash_bias_forward(q, k, v, qb, kb, None, False, 1.0 / math.sqrt(D), flags=flags)
    lib, stream, out = _lib.load(), torch.cuda.current_stream().cuda_stream, []
    for fused in (0, _lib.FB_FLAG_BWD_FUSED_DELTA):
        p = _lib.FbParams()
        _fill_common(p, q, k, v, qb, kb, None, False, float(sc), flags | fused)
        grads = [torch.empty_like(t) for t in (q, k, v, qb, kb)]
        delta = torch.full_like(lse, float("nan"))
        p.o, p.o_stride, p.lse, p.lse_stride_bh = o.data_ptr(), _strides_bhs(o), lse.data_ptr(), lse.shape[-1]
        p.dout, p.dout_stride, p.delta = do.data_ptr(), _strides_bhs(do), delta.data_ptr()
        for name, t in zip(("dq", "dk", "dv", "dq_bias", "dk_bias"), grads):
            setattr(p, name, t.data_ptr())
            setattr(p, name + "_stride", _strides_bhs(t))
        ws = torch.empty(lib.fb_bwd_workspace_bytes(C.byref(p)), dtype=torch.uint8, device="cuda")
        p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
        if not fused:
            assert lib.fb_bwd_preprocess(C.byref(p), stream) == 0
        assert lib.fb_bwd(C.byref(p), stream) == 0
        torch.cuda.synchronize()
        out.append((delta[..., :130], *grads))
    assert torch.equal(out[0][0], out[1][0])
    want = (o.float() * do.float()).sum(-1).permute(0, 2, 1)
    assert (out[1][0] - want).abs().max() <= 1e-4 * want.abs().max()
    for a, b in zip(out[0], out[1]):
        assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max()
