"""Build libtllm.so (the C-ABI shared library) in-tree with nvcc for sm_100a, and `_binding.so` (the CPython extension that
calls it from torch tensors) with g++.

    python -m ternaryllm_b200.build [--force] [--verbose]

The library has no dependency on torch; the extension has, and links the library from its own folder.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtllm.so")
SOURCES = ["capi.cu", "bits.cu", "comm.cu", "packer.cpp", "bstream_pack.cpp", "ssr_format.cpp"]
DEPS = ["kernels.cuh", "attn_kernel.cuh", "column_sum.cuh", "lists_kernel.cuh", "bits_kernel.cuh", "mma_kernel.cuh", "mma_units4_kernel.cuh", "bstream_kernel.cuh", "nibble_kernel.cuh", "nibble_rows_kernel.cuh", "nibble_format.h", "bstream_format.h", "bittile_format.h", "column_lists.h", "util.h", os.path.join("..", "..", "include", "tllm.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-O2", "--shared", "-Xptxas", "-v", "-t", "0",
]

BINDING = os.path.join(HERE, "_binding.so")
BINDING_DEPS = ["binding.cpp", os.path.join("..", "..", "include", "tllm.h")]


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in deps)


def _run(cmd, verbose: bool, log_mode: str) -> None:
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    log = os.path.join(HERE, "build.log")
    with open(log, log_mode) as f:
        f.write(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed; see " + log)
    if verbose:
        print(r.stdout)


def build_binding(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale(BINDING, BINDING_DEPS):
        return BINDING
    import sysconfig

    import torch

    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
           os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           os.path.join(CSRC, "binding.cpp")] + ["-I" + i for i in inc] + \
        ["-L" + HERE, "-l:libtllm.so", "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
         "-Wl,-rpath,$ORIGIN", "-o", BINDING]
    _run(cmd, verbose, "a")
    return BINDING


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _stale(LIB, SOURCES + DEPS):
        nvcc = os.environ.get("NVCC", "nvcc")
        _run([nvcc] + NVCC_FLAGS + [os.path.join(CSRC, s) for s in SOURCES] + ["-o", LIB], verbose, "w")
    build_binding(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
