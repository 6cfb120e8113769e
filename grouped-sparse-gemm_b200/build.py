"""Build libpaired_nvfp4_b200.so in-tree with nvcc for sm_100a (no torch dependency), then the operator layer
libpaired_nvfp4_torch.so (C++ against torch's headers) that registers torch.ops.paired_nvfp4.* on top of it.

    python grouped-sparse-gemm_b200/build.py [--force] [--ptxas-v]

Both land in grouped-sparse-gemm_b200/paired_nvfp4_kernels/, next to the Python package
that loads them.  PAIRED_NVFP4_PTXAS_V=1 (or --ptxas-v) prints registers / spills / shared memory.
"""
import os
import runpy
import subprocess
import sys
from importlib.util import find_spec

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "paired_nvfp4_kernels", "libpaired_nvfp4_b200.so")
TORCH_SRC = os.path.join(CSRC, "torch_ops.cpp")
TORCH_OUT = os.path.join(HERE, "paired_nvfp4_kernels", "libpaired_nvfp4_torch.so")
HEADER = os.path.join(os.path.dirname(HERE), "include", "paired_nvfp4_b200.h")
SOURCES = ["abi.cu", "quant.cu", "compress.cu", "routing.cu", "group_mm.cu"]


def _inputs():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))] + [HEADER]


def up_to_date(out, inputs):
    if not os.path.exists(out):
        return False
    t = os.path.getmtime(out)
    return all(os.path.getmtime(f) <= t for f in inputs)


def _run(cmd, verbose):
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)


def _cuda_home():
    return os.environ.get("CUDA_HOME", "/usr/local/cuda")


def build(force=False, ptxas_v=False, verbose=True):
    if force or not up_to_date(OUT, _inputs()):
        nvcc = os.environ.get("NVCC", os.path.join(_cuda_home(), "bin", "nvcc"))
        cmd = [nvcc, "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O3", "-lineinfo",
               "-gencode", "arch=compute_100a,code=sm_100a", "-o", OUT]
        if ptxas_v or os.environ.get("PAIRED_NVFP4_PTXAS_V") == "1":
            cmd += ["-Xptxas", "-v"]
        cmd += os.environ.get("PAIRED_NVFP4_NVCC_FLAGS", "").split()      # developer builds, e.g. -DPNV_WIDE_PROFILE
        _run(cmd + [os.path.join(CSRC, s) for s in SOURCES], verbose)
    build_torch_ops(force, verbose)
    return OUT


def torch_build_id():
    """Which torch an operator layer built now belongs to (read without importing torch).  C++ against torch's headers
    loads into that build alone."""
    version = runpy.run_path(os.path.join(os.path.dirname(find_spec("torch").origin), "version.py"))
    return f"torch-build:{version['__version__']}:{version.get('git_version')};"


def torch_ops_up_to_date():
    """Newer than its sources, and built for the torch that is installed: the library carries the id."""
    if not up_to_date(TORCH_OUT, [TORCH_SRC, HEADER]):
        return False
    with open(TORCH_OUT, "rb") as f:
        return torch_build_id().encode() in f.read()


def build_torch_ops(force=False, verbose=True):
    if not force and torch_ops_up_to_date():
        return TORCH_OUT
    import torch
    root = os.path.dirname(torch.__file__)
    lib = os.path.join(root, "lib")
    # the g++ on PATH, not $CXX: libstdc++ has to be the shared one that torch uses (a second, static copy inside this
    # library crashed while formatting an error message)
    _run(["g++", "-shared", "-fPIC", "-std=c++17", "-O2", "-fvisibility=hidden",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DPNV_TORCH_BUILD_ID="{torch_build_id()}"',
          "-isystem", os.path.join(root, "include"), "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
          "-isystem", os.path.join(_cuda_home(), "include"), TORCH_SRC, "-o", TORCH_OUT,
          "-L" + lib, "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
          "-L" + os.path.dirname(OUT), "-lpaired_nvfp4_b200", "-L" + os.path.join(_cuda_home(), "lib64"), "-lcudart",
          "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + lib], verbose)
    return TORCH_OUT


if __name__ == "__main__":
    build(force="--force" in sys.argv, ptxas_v="--ptxas-v" in sys.argv)
