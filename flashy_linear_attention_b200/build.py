"""Builds libflashlinear_sm100.so in-tree with nvcc for sm_100a, and _hostcalls.*.so beside it.

Usage: python -m flashy_linear_attention_b200.build [--force]
The library has no Python or torch dependency; it links the static CUDA runtime only. _hostcalls.*.so
is the host side of a call on torch tensors (csrc/fla_host.cpp), a Python extension on top of it that
needs g++. It is bound to one torch and one Python, so its name carries both versions: after an
upgrade it counts as missing, calls go through ctypes (same kernels, more host time) and say so once,
until this module has run again.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_NAME = "libflashlinear_sm100.so"
LIB_PATH = os.path.join(HERE, LIB_NAME)

SOURCES = ["fla_api.cu"]
HOST_SOURCES = ["fla_host.cpp", os.path.join("..", "..", "include", "flashlinear_sm100.h")]
HEADERS = ["fla_kernel.cuh", "fla_backward.cuh", "fla_wide_kernel.cuh", "fla_normalize.cuh", "fla_taylor.cuh", "fla_taylor_attention.cuh", "fla_decode.cuh", "ptx.cuh", os.path.join("..", "..", "include", "flashlinear_sm100.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
    "-cudart", "static",
]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build " + LIB_NAME)
    return nvcc


def host_path() -> str:
    """Where the extension for the running Python and the installed torch is built."""
    import torch

    return os.path.join(HERE, f"_hostcalls.torch-{torch.__version__}{sysconfig.get_config_var('EXT_SUFFIX')}")


def _stale(built_path: str, sources) -> bool:
    if not os.path.exists(built_path):
        return True
    built = os.path.getmtime(built_path)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > built for f in sources)


def is_stale() -> bool:
    return _stale(LIB_PATH, SOURCES + HEADERS) or _stale(host_path(), HOST_SOURCES)


def _run(cmd, what: str) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + res.stdout + res.stderr)
    return res.stderr


def build_host(force: bool = False) -> str:
    """Compiles the Python extension (host code only; links the library, found beside it)."""
    path = host_path()
    if not force and not _stale(path, HOST_SOURCES):
        return path
    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    cuda_home = os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc())))
    includes = include_paths() + [os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    cmd += [f"-I{p}" for p in includes]
    cmd += [os.path.join(CSRC, HOST_SOURCES[0]), "-o", path]
    cmd += [f"-L{p}" for p in library_paths()]
    cmd += [f"-L{HERE}", "-l:" + LIB_NAME, "-Wl,-rpath,$ORIGIN"]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python"]
    _run(cmd, "g++")
    return path


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles whatever is missing or older than its sources."""
    if force or _stale(LIB_PATH, SOURCES + HEADERS):
        cmd = [find_nvcc()] + NVCC_FLAGS
        if verbose:
            cmd += ["-Xptxas", "-v"]
        cmd += ["-o", LIB_PATH] + [os.path.join(CSRC, s) for s in SOURCES]
        out = _run(cmd, "nvcc")
        if verbose:
            print(out)
    build_host(force)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
