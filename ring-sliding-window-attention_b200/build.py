"""Builds ring_swa/librswa.so (the C-ABI library of include/rswa.h) with nvcc for sm_100a, and
ring_swa/_native.so (the C++ host path of a single-GPU call, linked to it and to torch) with g++.

    python ring-sliding-window-attention_b200/build.py [--force] [--verbose]

Both are built in-tree, next to the Python package that loads them.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "ring_swa", "librswa.so")
NATIVE_OUT = os.path.join(HERE, "ring_swa", "_native.so")
NATIVE_STAMP = NATIVE_OUT + ".stamp"
NATIVE_SOURCE = os.path.join(CSRC, "rswa_torch.cpp")
SOURCES = ["rswa_api.cu", "rswa_fwd.cu", "rswa_bwd.cu", "rswa_dq.cu", "rswa_aux.cu", "rswa_selftest.cu", "rswa_noalloc.cu", "rswa_peer.cu"]
HEADERS = ["tc05.cuh", "rswa_common.cuh", "rswa_tiles.cuh", os.path.join("..", "..", "include", "rswa.h")]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC")


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def is_stale() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = sources() + [os.path.join(CSRC, h) for h in HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _native_abi() -> str:
    """What _native.so is bound to besides its source: it includes torch's and Python's headers."""
    import torch
    return f"torch {torch.__version__} cxx11 {int(torch._C._GLIBCXX_USE_CXX11_ABI)} {sys.implementation.cache_tag}"


def native_is_stale() -> bool:
    if not os.path.exists(NATIVE_OUT) or not os.path.exists(NATIVE_STAMP):
        return True
    with open(NATIVE_STAMP) as f:
        if f.read() != _native_abi():
            return True
    deps = [NATIVE_SOURCE, os.path.join(CSRC, "..", "..", "include", "rswa.h"), os.path.abspath(__file__)]
    return os.path.getmtime(NATIVE_OUT) <= max(os.path.getmtime(d) for d in deps)


def build_native(force: bool = False) -> str:
    """The torch-facing host path; needs librswa.so, whose directory it looks in at load time."""
    if not force and not native_is_stale():
        return NATIVE_OUT
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    cmd = ["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-fvisibility=hidden", "-o", NATIVE_OUT, NATIVE_SOURCE,
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(cuda, "include"),
           "-L", os.path.join(HERE, "ring_swa"), "-l:librswa.so", "-Wl,-rpath,$ORIGIN",
           "-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
    with open(NATIVE_STAMP, "w") as f:
        f.write(_native_abi())
    return NATIVE_OUT


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not is_stale():
        build_native()
        return OUT
    cmd = [
        _nvcc(), "-std=c++17", "-O3", "-lineinfo",
        "-gencode", "arch=compute_100a,code=sm_100a",
        "-shared", "-Xcompiler", "-fPIC",
        "-o", OUT,
    ]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += sources()
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stdout + res.stderr)
    build_native(force)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
