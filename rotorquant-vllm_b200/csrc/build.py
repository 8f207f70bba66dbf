"""Build librq_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and ``_host-<torch>.so``,
the native side of the Python launchers, with the host compiler against the installed torch.

Usage: ``python rotorquant-vllm_b200/csrc/build.py [--verbose]``.  Both are written next to the
Python package that loads them (``rotorquant-vllm_b200/rotorquant_vllm/``).
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

CSRC = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(CSRC), "rotorquant_vllm")
LIB = os.path.join(PKG, "librq_b200.so")
HOST_SOURCE = os.path.join(CSRC, "rq_host.cpp")
SOURCES = ["rq_api.cu", "rq_compress.cu", "rq_decode.cu", "rq_peer.cu", "rq_prefill.cu", "rq_probe.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; librq_b200.so cannot be built")
    return exe


def _stale(lib: str) -> bool:
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".cpp"))]
    deps.append(os.path.join(os.path.dirname(os.path.dirname(CSRC)), "include", "rq_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def host_library() -> str:
    """Path of the launchers' native side for this interpreter and the installed torch: another torch
    asks for another file, so that a module is never loaded into one that it was not built against."""
    import torch

    return os.path.join(PKG, f"_host-{sys.implementation.cache_tag}-torch{torch.__version__}.so")


def build_host(force: bool = False) -> str:
    """Compile the native side of the launchers (a CPython extension module); returns its path."""
    lib = host_library()
    if not force and not _stale(lib):
        return lib
    from torch._C import _GLIBCXX_USE_CXX11_ABI
    from torch.utils.cpp_extension import include_paths, library_paths

    includes = [f"-I{d}" for d in [*include_paths("cuda"), sysconfig.get_paths()["include"]]]
    dirs = [flag for d in library_paths("cuda") for flag in (f"-L{d}", f"-Wl,-rpath,{d}")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(_GLIBCXX_USE_CXX11_ABI)}", *includes, HOST_SOURCE, "-o", lib, *dirs,
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-lcudart"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(" ".join(cmd) + "\n" + proc.stdout + proc.stderr)
    return lib


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``.cu`` file into one shared library, and the launchers' native side; returns
    the path of the former."""
    srcs = [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    build_host(force)
    if not force and not _stale(LIB):
        return LIB
    cmd = [_nvcc(), "-O3", "-std=c++17", *ARCH, "-lineinfo", "--shared", "-Xcompiler", "-fPIC",
           "--threads", "0", "-o", LIB, *srcs]
    if verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + proc.stdout + proc.stderr)
    if verbose:
        print(proc.stderr)
    return LIB


if __name__ == "__main__":
    print(build_library(force=True, verbose="--verbose" in sys.argv))
