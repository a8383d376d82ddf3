"""Build libflashbias_b200.so in-tree with nvcc for sm_100a.

    python -m flashbias_b200.build [--force] [--verbose]
    python flashbias_b200/build.py        (the same, without importing the package)

The C library needs nvcc alone.  The PyTorch extension with the operators' host path is built beside it where torch is
installed; without torch the C library is all there is.

The shared library lands next to the package (``flashbias_b200/libflashbias_b200.so``) so that it
travels with the source tree; nothing is installed into site-packages and nothing is JIT-cached.
"""
from __future__ import annotations

import hashlib
import os
import re
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libflashbias_b200.so")
TORCH_OP = os.path.join(PKG, "_torch_op.so")  # the operators' host path (csrc/torch_op.cpp), linked against LIB

SOURCES = ["fb_api.cu", "fb_tmap.cu", "fb_pack.cu", "fb_finish.cu", "fb_general.cu", "fb_selftest.cu",
           "fb_fwd_sm100.cu", "fb_fwd_inst_d32.cu", "fb_fwd_inst_d64.cu", "fb_fwd_inst_d128.cu", "fb_fwd_inst_s128.cu",
           "fb_bwd_sm100.cu", "fb_bwd_inst_d32.cu", "fb_bwd_inst_d32p.cu", "fb_bwd_inst_d64.cu", "fb_bwd_inst_d128.cu", "fb_bwd_inst_s32.cu", "fb_bwd_inst_s64.cu",
           "fb_decode.cu", "fb_noalloc.cu", "fb_prepare.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--use_fast_math", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I", CSRC]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add the CUDA toolkit to PATH")


def _build_torch_op(verbose: bool) -> None:
    """The PyTorch extension with the operators' host path; a CPU compile against the installed torch headers."""
    import sysconfig

    from torch.utils import cpp_extension
    inc = [os.path.join(ROOT, "include"), sysconfig.get_paths()["include"], "/usr/local/cuda/include",
           *cpp_extension.include_paths()]
    libdirs = cpp_extension.library_paths()
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_torch_op",
           *[x for i in inc for x in ("-isystem", i)], os.path.join(CSRC, "torch_op.cpp"), "-o", TORCH_OP,
           LIB, "-Wl,-rpath,$ORIGIN", *[f"-L{d}" for d in libdirs],
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on torch_op.cpp:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)


def _torch_version() -> str | None:
    try:
        import torch
    except ImportError:
        return None
    return torch.__version__


def _digest(paths, salt: str = "") -> str:
    h = hashlib.sha256(salt.encode())
    for p in sorted(paths):
        with open(p, "rb") as f:
            h.update(p.encode() + b"\0" + f.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def _with_headers(path, seen=None):
    """The source file and, transitively, the headers of this project it includes."""
    seen = set() if seen is None else seen
    if path in seen:
        return seen
    seen.add(path)
    with open(path) as f:
        for name in re.findall(r'^\s*#include "([^"]+)"', f.read(), flags=re.M):
            for d in (CSRC, os.path.join(ROOT, "include")):
                if os.path.exists(os.path.join(d, name)):
                    _with_headers(os.path.join(d, name), seen)
    return seen


def build(force: bool = False, verbose: bool = False) -> str:
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(ROOT, "include", "flashbias_b200.h"))
    os.makedirs(OBJ, exist_ok=True)
    stamp, op_stamp = os.path.join(OBJ, "stamp"), os.path.join(OBJ, "torch_op.stamp")
    digest = _digest([os.path.join(CSRC, s) for s in srcs] + headers)
    torch_version = _torch_version()
    op_digest = torch_version and _digest(_with_headers(os.path.join(CSRC, "torch_op.cpp")), torch_version)

    def is_current(target, stamp_path, want):
        return not force and os.path.exists(target) and os.path.exists(stamp_path) and open(stamp_path).read() == want

    if not is_current(LIB, stamp, digest):
        _build_library(srcs, force, verbose)
        with open(stamp, "w") as f:
            f.write(digest)
    if op_digest and not is_current(TORCH_OP, op_stamp, op_digest):
        _build_torch_op(verbose)
        with open(op_stamp, "w") as f:
            f.write(op_digest)
    return LIB


def _build_library(srcs, force: bool, verbose: bool) -> None:
    nvcc = _nvcc()
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src):
        obj = os.path.join(OBJ, src.replace(".cu", ".o"))
        # per-object stamp over the source and the headers it includes: only what changed is compiled again
        own, done = _digest(_with_headers(os.path.join(CSRC, src))), obj + ".stamp"
        if not force and not verbose and os.path.exists(obj) and os.path.exists(done) and open(done).read() == own:
            return obj
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        with open(done, "w") as f:
            f.write(own)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    r = subprocess.run([nvcc, "-shared", "-o", LIB, "-Xlinker", "-soname=libflashbias_b200.so", *objs, "-gencode", "arch=compute_100a,code=sm_100a"],
                       capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
