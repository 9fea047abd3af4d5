"""Builds the two native libraries in-tree: libegs_b200.so (kernels behind the C ABI, nvcc for sm_100a) and _egs_host.so (the
host path: operators, autograd functions and the training step over that ABI, g++ against the installed torch).

    python -m expertscattergather_b200.build [--force] [--verbose]

Both are written to ``expertscattergather_b200/_lib/`` and rebuilt when a source file is newer.  No GPU is needed.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OUT_DIR = os.path.join(PKG, "_lib")
OBJ_DIR = os.path.join(OUT_DIR, "obj")
LIB_PATH = os.path.join(OUT_DIR, "libegs_b200.so")
HOST_PATH = os.path.join(OUT_DIR, "_egs_host.so")
SOURCES = ["egs_api.cu", "egs_generic.cu", "egs_tensor.cu", "egs_strict.cu", "egs_dense16.cu", "egs_pair16.cu", "egs_gather2.cu", "egs_index.cu"]
HOST_SOURCE = os.path.join(CSRC, "egs_host.cpp")
API_HEADER = os.path.join(PKG, "..", "include", "egs_b200.h")
HEADERS = [os.path.join(CSRC, "egs_internal.cuh"), os.path.join(CSRC, "egs_tcgen05.cuh"), API_HEADER]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC or put it on PATH)")


def _newer(target: str, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def needs_build() -> bool:
    return _newer(LIB_PATH, [os.path.join(CSRC, s) for s in SOURCES] + HEADERS)


def host_needs_build() -> bool:
    return _newer(HOST_PATH, [HOST_SOURCE, API_HEADER])


def _run(cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed building {cmd[cmd.index('-o') + 1]}")


def _build_kernels(force: bool, verbose: bool) -> None:
    os.makedirs(OBJ_DIR, exist_ok=True)
    flags = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
             "-Xcompiler", "-O2"] + (["-Xptxas", "-v"] if verbose else [])
    objs, jobs = [], []
    with concurrent.futures.ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        for s in SOURCES:
            src, obj = os.path.join(CSRC, s), os.path.join(OBJ_DIR, s + ".o")
            objs.append(obj)
            if force or _newer(obj, [src] + HEADERS):
                jobs.append(pool.submit(_run, flags + ["-c", src, "-o", obj], verbose))
        for j in jobs:
            j.result()
    _run(flags + ["-shared"] + objs + ["-o", LIB_PATH, "-lcudart"], False)


def _build_host(verbose: bool) -> None:
    import torch
    from torch.utils import cpp_extension
    os.makedirs(OUT_DIR, exist_ok=True)
    cuda_home = os.path.dirname(os.path.dirname(_nvcc()))
    incs = cpp_extension.include_paths() + [os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    lib_dirs = cpp_extension.library_paths() + [os.path.join(cuda_home, "lib64")]
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_egs_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    cmd += [f for d in incs for f in ("-isystem", d)] + [HOST_SOURCE, "-o", HOST_PATH]
    cmd += [f"-L{d}" for d in lib_dirs] + [f"-Wl,-rpath,{d}" for d in lib_dirs[:1]]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lcudart", "-ldl"]
    _run(cmd, verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Builds what is out of date; returns the path of the kernel library."""
    kernels, host = force or needs_build(), force or host_needs_build()
    with concurrent.futures.ThreadPoolExecutor(max_workers=2) as pool:
        jobs = ([pool.submit(_build_kernels, force, verbose)] if kernels else []) + ([pool.submit(_build_host, verbose)] if host else [])
        for j in jobs:
            j.result()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
