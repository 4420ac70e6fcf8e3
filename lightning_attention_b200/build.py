"""Builds liblightning_b200.so (the C-ABI library with all sm_100a kernels) in-tree with nvcc, and beside it _host_ops.so (the
operators' native call path, a CPython extension on torch's C++ API; no device code) with g++.

Run as ``python -m lightning_attention_b200.build``. Cross-compiles without a GPU.
"""
import os
import shutil
import subprocess
import sys

if __package__:
    from . import _lib
else:  # run by its path
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    from lightning_attention_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_NAME = "liblightning_b200.so"
LIB_PATH = os.path.join(HERE, LIB_NAME)
SOURCES = [os.path.join(HERE, "csrc", "capi.cu")]
import glob

HEADERS = sorted(glob.glob(os.path.join(HERE, "csrc", "*.cuh"))) + [os.path.join(HERE, "..", "include", "lightning_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


HOST_PATH = _lib.HOST_PATH
HOST_SOURCES = [os.path.join(HERE, "csrc", "host_ops.cpp"), os.path.join(HERE, "..", "include", "lightning_b200.h")]


def find_nvcc():
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
        if os.path.exists(cand):
            nvcc = cand
    if nvcc is None:
        raise RuntimeError("nvcc not found; cannot build " + LIB_NAME)
    return nvcc


def _newer(path, sources):
    if not os.path.exists(path):
        return False
    t = os.path.getmtime(path)
    return all(os.path.getmtime(f) <= t for f in sources if os.path.exists(f))


def _run(cmd, what, verbose):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + res.stdout + res.stderr)


def build_host(verbose=False):
    """Compile _host_ops.so against the torch this interpreter imports."""
    import sysconfig

    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(find_nvcc()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DLAB200_HOST_ABI="{_lib.host_abi()}"']
    cmd += [a for d in inc for a in ("-isystem", d)] + ["-o", HOST_PATH, HOST_SOURCES[0], "-L" + os.path.join(root, "lib")]
    _run(cmd + ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python"], "g++", verbose)
    return HOST_PATH


def build(force=False, verbose=False):
    """Compile what is missing or older than its sources. Returns the path of the C-ABI library."""
    if force or not _newer(LIB_PATH, SOURCES + HEADERS):
        _run([find_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] + SOURCES, "nvcc", verbose)
    if force or not _newer(HOST_PATH, HOST_SOURCES) or _lib.host_built_for(HOST_PATH) != _lib.host_abi():
        build_host(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
