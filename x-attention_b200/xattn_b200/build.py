"""Compile csrc/*.cu into libxattn_b200.so (sm_100a) and csrc/host_ops.cpp into _host.so, next to this file.

    python -m xattn_b200.build [--force]

nvcc cross-compiles without a GPU.  The library has no torch dependency (it is also loaded with ctypes); _host.so is the
CPython module that calls it on torch tensors.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libxattn_b200.so")
HOST = os.path.join(HERE, "_host.so")
HEADER = os.path.join(os.path.dirname(os.path.dirname(HERE)), "include", "xattn_b200.h")
SOURCES = ["api.cu", "estimate.cu", "estimate_noalloc.cu", "select.cu", "attention.cu", "attention_pair.cu",
           "decode.cu", "rope.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared", "-diag-suppress", "550"]


def _stale(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in sources if os.path.exists(d))


def _run(cmd, what: str, verbose: bool) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(what + " failed:\n" + r.stdout + r.stderr)
    if verbose:
        print(r.stdout + r.stderr)


def build_host(force: bool = False, verbose: bool = False) -> str:
    """The tensor plumbing as a CPython module against the installed torch, linked to libxattn_b200.so."""
    src = os.path.join(CSRC, "host_ops.cpp")
    if not force and not _stale(HOST, [src, HEADER, LIB]):
        return HOST
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        raise RuntimeError("no C++ compiler found: cannot build _host.so")
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for i in inc:
        cmd += ["-isystem", i]
    cmd += [src, "-o", HOST, "-L" + HERE, "-l:libxattn_b200.so", "-Wl,-rpath,$ORIGIN", "-L" + os.path.join(root, "lib"),
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    _run(cmd, "g++", verbose)
    return HOST


def build(force: bool = False, verbose: bool = False) -> str:
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))] + [HEADER]
    if force or _stale(LIB, deps):
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not os.path.exists(nvcc):
            raise RuntimeError("nvcc not found: cannot build libxattn_b200.so")
        cmd = [nvcc, *NVCC_FLAGS, "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        _run(cmd, "nvcc", verbose)
    build_host(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
