"""Builds libdn_cuda.so in-tree for sm_100a (B200).

    python -m ding_nsch_core_solver_b200.build

nvcc cross-compiles without a GPU.  The library is compiled with --fmad=false: the stencil kernels keep
the reference's operand order and then round exactly like it; hot loops use explicit fma where wanted.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libdn_cuda.so")
SOURCES = ["dn_capi.cu", "dn_config.cpp"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
# No -split-compile: with it the kernels' code depends on how many cores the building machine has (one source gave
# k_bicgstab 127 or 64 registers and k_wpcg 156 or 124; the 512 x 1024 pressure solve took 233 or 251 ms and other bits).
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "--fmad=false", "-std=c++17",
         "-Xcompiler", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "include")]


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", "dn_cuda.h"),
                                                                  os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    cmd = [NVCC] + FLAGS + [os.path.join(CSRC, s) for s in SOURCES] + ["-o", LIB]
    if verbose:
        print(" ".join(cmd))
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
