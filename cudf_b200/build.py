"""In-tree build of the CUDA library (sm_100a only) and of the CPython extension over it.

``python -m cudf_b200.build`` compiles cudf_b200/csrc/b2_groupby.cu into
cudf_b200/libb2groupby.so with nvcc (which cross-compiles without a GPU), and
cudf_b200/csrc/b2_native.cpp, which links to it and to torch, into cudf_b200/_b2native.so with g++.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc", "b2_groupby.cu")
DEPS = [SRC, os.path.join(HERE, "csrc", "b2_kernels.cuh"), os.path.join(HERE, "csrc", "b2_box.cuh"), os.path.join(HERE, "csrc", "b2_lean.cuh"), os.path.join(HERE, "csrc", "b2_partition.cuh"), os.path.join(HERE, "csrc", "b2_keyed.cuh"),
        os.path.join(HERE, "csrc", "b2_device.cuh"),
        os.path.join(os.path.dirname(HERE), "include", "b2_groupby.h")]
LIB = os.path.join(HERE, "libb2groupby.so")
NATIVE_SRC = os.path.join(HERE, "csrc", "b2_native.cpp")
NATIVE_DEPS = [NATIVE_SRC, os.path.join(os.path.dirname(HERE), "include", "b2_groupby.h")]
NATIVE = os.path.join(HERE, "_b2native.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared", "-cudart", "shared", "-ldl"]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return nvcc


def _older(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in sources)


def stale() -> bool:
    return _older(LIB, DEPS) or _older(NATIVE, NATIVE_DEPS)


def _run(cmd, verbose: bool):
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + proc.stdout + proc.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    """Builds libb2groupby.so and _b2native.so where they are missing or older than their sources; returns the
    library's path."""
    if force or _older(LIB, DEPS):
        _run([find_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB, SRC], verbose)
    if force or _older(NATIVE, NATIVE_DEPS):
        import torch
        root = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc())))
        inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
        _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] +
             [f"-I{i}" for i in inc] + ["-o", NATIVE, NATIVE_SRC, f"-L{HERE}", "-l:libb2groupby.so", "-Wl,-rpath,$ORIGIN",
             "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"], verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
