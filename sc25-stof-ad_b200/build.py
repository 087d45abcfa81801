"""Builds libstof_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _stof_native.so (the host path of the Python
operators, against torch's headers) with g++.

    python sc25-stof-ad_b200/build.py [--verbose] [--force]

The library links the CUDA runtime statically and resolves the one driver entry point it
needs (tensor-map encoding) at run time, so it also loads on a machine without a GPU.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "stof_b200", "libstof_b200.so")
NATIVE_SRC = os.path.join(CSRC, "host", "stof_native.cpp")
NATIVE = os.path.join(HERE, "stof_b200", "_stof_native.so")

NVCC_FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC"]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _native_command():
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-I" + sysconfig.get_paths()["include"],
            "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I" + os.path.join(cuda, "include"), NATIVE_SRC, "-o", NATIVE, "-L" + os.path.join(root, "lib"),
            "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(NATIVE):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(NATIVE))
    deps = [NATIVE_SRC] + sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h")) + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(verbose: bool = False, force: bool = False) -> str:
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    for src in sources():
        obj = os.path.splitext(src)[0] + ".o"
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    procs.append((NATIVE_SRC, subprocess.Popen(_native_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stderr.write(out)
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("compilation failed")
    subprocess.check_call([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs, "-cudart", "static", "-Xcompiler", "-fPIC"])
    return LIB


if __name__ == "__main__":
    print(build_library(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
