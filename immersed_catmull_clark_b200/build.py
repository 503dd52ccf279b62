"""Build recipe for libicc.so (the C-ABI library) for sm_100a, in-tree.

    python -m immersed_catmull_clark_b200.build
"""
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libicc.so")
SOURCES = ["icc_op.cu", "icc_modal.cu", "icc_mixed.cu", "icc_topopt.cu", "icc_immersed.cu", "icc_noalloc.cu", "icc_space.cpp", "icc_stab.cpp"]
HEADERS = ["icc_internal.h", "icc_device.cuh", "icc_vec.cuh", "icc_modal.cuh", "icc_tc.cuh"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-diag-error", "2809",            # a dropped launch status ([[nodiscard]]) fails the build
    "-Xcompiler", "-fPIC", "-shared",
    "-I", os.path.join(ROOT, "include"),
]


def needs_build():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(ROOT, "include", "icc.h")]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB
    cmd = ["nvcc"] + NVCC_FLAGS + ["-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
        print(" ".join(cmd))
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    build(force=True, verbose="-v" in sys.argv)
    print(LIB)
