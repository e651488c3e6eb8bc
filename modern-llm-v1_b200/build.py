"""Builds the native code in-tree: csrc/b200attn_api.cu -> libb200attn.so (CUDA, sm_100a only) and
csrc/host_binding.cc -> _host.so (the Python module over its C ABI).

nvcc cross-compiles without a GPU, so this also runs on a CPU-only machine.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200attn.so")
HOST = os.path.join(HERE, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-shared", "-Xcompiler", "-fPIC",
]


def sources() -> list[str]:
    out = []
    for root, _, files in os.walk(CSRC):
        for f in files:
            if f.endswith((".cu", ".cuh", ".h", ".cc")):
                out.append(os.path.join(root, f))
    out.append(os.path.join(os.path.dirname(HERE), "include", "b200attn.h"))
    return out


def is_stale() -> bool:
    if not (os.path.exists(LIB) and os.path.exists(HOST)):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST))
    return any(os.path.getmtime(s) > t for s in sources())


def _host_command() -> list[str]:
    import sysconfig

    import torch

    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"))
    inc = [os.path.join(t, "include"), os.path.join(t, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    # torch's libraries are in the process by the time the module is imported; libb200attn.so lies beside it
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={abi}",
            *(f"-I{i}" for i in inc), "-o", HOST, os.path.join(CSRC, "host_binding.cc"), f"-L{HERE}", "-l:libb200attn.so",
            f"-L{os.path.join(t, 'lib')}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles both libraries if one is missing or older than the sources; returns the CUDA library's path."""
    if not force and not is_stale():
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    cmd = [nvcc, *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB, os.path.join(CSRC, "b200attn_api.cu")]
    subprocess.check_call(cmd)
    subprocess.check_call(_host_command())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
