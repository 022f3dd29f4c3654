"""Ahead-of-time build of lib/libb200fp8mm.so with nvcc for sm_100a.

Replaces the reference's import-time JIT (`load_inline` with hipcc for gfx942,
1-amd-fp8-mm/amd-fp8-mm-submission.py:582-592)."""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
INCLUDE = os.path.join(ROOT, "include")
SRC = os.path.join(HERE, "csrc", "fp8_mm_sm100.cu")
SOURCES = [SRC, os.path.join(HERE, "csrc", "mla_consumers_sm100.cu")]
HEADERS = [os.path.join(INCLUDE, "b200_fp8_mm.h"), os.path.join(INCLUDE, "b200_mla_consumers.h"),
           os.path.join(HERE, "csrc", "issuer_walk.h")]
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libb200fp8mm.so")
HOST_SRC = os.path.join(HERE, "csrc", "host_calls.cpp")  # the entry points' per-call host work (a CPython module)


def host_path() -> str:
    """Where the native module for the running Python and torch lies. It is compiled against the internals of both, so both
    are in its name and a module built for others is neither loaded nor taken for up to date."""
    import sysconfig

    import torch

    return os.path.join(LIB_DIR, f"_host.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so")


def _nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _outdated(target: str, sources) -> bool:
    return not os.path.exists(target) or os.path.getmtime(target) < max(os.path.getmtime(p) for p in sources)


def needs_build() -> bool:
    return _outdated(LIB, SOURCES + HEADERS) or _outdated(host_path(), [HOST_SRC] + HEADERS)


def _build_host() -> None:
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    includes = [INCLUDE, sysconfig.get_paths()["include"], *include_paths("cuda")]
    subprocess.check_call([
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *(f"-I{p}" for p in includes),
        HOST_SRC, "-o", host_path(), *(f"-L{p}" for p in library_paths()),
        "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python",
    ])


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    if force or _outdated(host_path(), [HOST_SRC] + HEADERS):
        _build_host()
    if not force and not _outdated(LIB, SOURCES + HEADERS):
        return LIB
    cmd = [
        _nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
        "-I", INCLUDE, "-shared", "-Xcompiler", "-fPIC", "-o", LIB, *SOURCES,
    ]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
