"""The C-ABI library loads, exports every symbol the public header declares, and rejects bad
arguments on the host before touching a device (no compute calls here)."""
import ctypes as C
import os
import re

import pytest

from flashbias_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_functions():
    text = open(os.path.join(ROOT, "include", "flashbias_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(fb_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    lib = _lib.load()
    names = _declared_functions()
    assert "fb_fwd" in names and "fb_bwd" in names and "fb_bwd_preprocess" in names
    for n in names:
        assert hasattr(lib, n), f"{n} declared in the header but not exported"
    assert set(names) == set(_lib.EXPORTS), "binding table and header disagree"


def test_struct_mirror_matches():
    assert _lib.load().fb_params_size() == C.sizeof(_lib.FbParams)


def _valid_params():
    p = _lib.FbParams()
    p.B, p.H, p.Sq, p.Sk, p.D, p.R = 1, 2, 128, 128, 32, 0
    p.dtype = _lib.FB_DTYPE_BF16
    p.softmax_scale = 0.25
    for name in ("q", "k", "v", "o", "lse"):
        setattr(p, name, 0x1000)  # never dereferenced on the host
    for name in ("q_stride", "k_stride", "v_stride", "o_stride"):
        setattr(p, name, _lib.I64x3(128 * 64, 32, 64))
    p.lse_stride_bh = 128
    return p


@pytest.mark.parametrize("mutate,code", [
    (lambda p: setattr(p, "q", None), -1),
    (lambda p: setattr(p, "D", 129), -2),
    (lambda p: setattr(p, "Sq", 0), -2),
    (lambda p: setattr(p, "dtype", 2), -3),
    (lambda p: setattr(p, "q_stride", _lib.I64x3(-1, 32, 64)), -4),
    (lambda p: setattr(p, "mask_kind", 1), -5),
    (lambda p: setattr(p, "R", 4), -7),
    (lambda p: setattr(p, "lse_stride_bh", 64), -8),
])
def test_host_side_validation(mutate, code):
    lib = _lib.load()
    p = _valid_params()
    mutate(p)
    assert lib.fb_fwd(C.byref(p), None) == code
    assert _lib.strerror(code)


def _problem(D=32, Sq=256, R=0, dtype=_lib.FB_DTYPE_BF16, scale=None, flags=0, slopes=False, mask=False, odd=False):
    p = _valid_params()
    p.D, p.Sq, p.Sk, p.R, p.dtype, p.flags = D, Sq, 256, R, dtype, flags
    p.softmax_scale = scale or D ** -0.5
    row = 2 * D + (1 if odd else 0)
    for name in ("q_stride", "k_stride", "v_stride", "o_stride"):
        setattr(p, name, _lib.I64x3(256 * row, D, row))
    p.lse_stride_bh = 256
    if R:
        p.q_bias = p.k_bias = 0x1000
        p.q_bias_stride = p.k_bias_stride = _lib.I64x3(0, R, 2 * R)
    if slopes:
        p.alibi_slopes = 0x1000
    if mask:
        p.mask, p.mask_kind, p.mask_dtype = 0x1000, _lib.FB_MASK_VECTOR, _lib.FB_DTYPE_F32
    return p


@pytest.mark.parametrize("problem,fwd,bwd", [
    (dict(R=2), "fwd_tiled", "bwd_two_stream"),
    (dict(R=2, flags=_lib.FB_FLAG_BWD_PERSISTENT), "fwd_tiled", "bwd_persistent"),
    (dict(R=2, flags=_lib.FB_FLAG_BWD_PERSISTENT | _lib.FB_FLAG_BWD_ONE_ITEM), "fwd_tiled", "bwd_query_major"),
    (dict(R=2, mask=True), "fwd_tiled", "bwd_query_major"),
    (dict(slopes=True), "fwd_tiled", "bwd_two_stream"),
    (dict(mask=True), "fwd_tiled", "bwd_key_major"),
    (dict(slopes=True, flags=_lib.FB_FLAG_BWD_QUERY_MAJOR), "fwd_tiled", "bwd_query_major"),
    (dict(mask=True, flags=_lib.FB_FLAG_BWD_QUERY_MAJOR), "fwd_tiled", "bwd_query_major"),
    (dict(D=64), "fwd_tiled", "bwd_two_stream"),
    (dict(D=64, R=8), "fwd_tiled", "bwd_two_stream"),
    (dict(D=64, R=9, scale=0.125), "fwd_tiled", "bwd_query_major"),
    (dict(D=64, mask=True), "fwd_tiled", "bwd_query_major"),
    (dict(D=72), "fwd_two_stream", "bwd_key_major"),
    (dict(D=128, slopes=True), "fwd_two_stream", "bwd_key_major"),
    (dict(D=128, mask=True), "fwd_tiled", "bwd_key_major"),
    (dict(D=128, R=32), "fwd_two_stream", "general"),
    (dict(D=128, R=33), "fwd_tiled", "general"),
    (dict(D=128, R=2), "fwd_two_stream", "general"),
    (dict(D=64, R=12, dtype=_lib.FB_DTYPE_F16), "fwd_tiled", "general"),
    (dict(R=40), "fwd_tiled", "general"),
    (dict(R=130), "general", "general"),
    (dict(D=20), "general", "general"),
    (dict(odd=True), "general", "general"),
    (dict(slopes=True, mask=True), "general", "general"),
    (dict(flags=_lib.FB_FLAG_FORCE_GENERAL), "general", "general"),
    (dict(Sq=1), "fwd_one_query", "bwd_two_stream"),
    (dict(Sq=1, slopes=True, mask=True), "fwd_one_query", "general"),
    (dict(Sq=1, R=17), "fwd_tiled", "bwd_two_stream"),
    (dict(Sq=1, scale=-1.0), "fwd_one_query", "general"),
    (dict(scale=-1.0), "general", "general"),
], ids=str)
def test_kernel_queries_name_the_kernel_taken(problem, fwd, bwd):
    lib, p = _lib.load(), _problem(**problem)
    assert _lib.KERNELS[lib.fb_fwd_kernel(C.byref(p))] == fwd
    assert _lib.KERNELS[lib.fb_bwd_kernel(C.byref(p))] == bwd


def test_kernel_queries_reject_what_the_launches_reject():
    lib, p = _lib.load(), _problem(D=129)
    assert lib.fb_fwd_kernel(C.byref(p)) == lib.fb_bwd_kernel(C.byref(p)) == -2


def test_backward_requires_gradient_buffers():
    lib = _lib.load()
    p = _valid_params()
    assert lib.fb_bwd(C.byref(p), None) == -1
    assert lib.fb_bwd_preprocess(C.byref(p), None) == -1


def test_missing_library_fails_loudly(monkeypatch):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", "/nonexistent/libflashbias_b200.so")
    with pytest.raises(RuntimeError, match="no fallback"):
        _lib.load()
