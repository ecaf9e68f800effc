"""Compiles libfrx.so (every CUDA source under csrc/) for sm_100a, in tree, and _frxpy.so, the Python
binding of its frequently called entry points.

    python -m flashrt_b200.build

nvcc cross-compiles without a GPU. The library is the product: the Python layer only binds it.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB = os.path.join(HERE, "libfrx.so")
BINDING = os.path.join(HERE, "_frxpy.so")


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(HERE, "csrc", "*.cu")))


def needs_build() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(BINDING):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(BINDING))
    deps = sources() + glob.glob(os.path.join(HERE, "csrc", "*.c")) + glob.glob(os.path.join(HERE, "csrc", "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "-Xfatbin", "-compress-all",   # (nvcc compresses device code of its own accord only above some size)
           "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(HERE, "csrc"),
           "-shared", "-Xcompiler", "-fPIC", "-o", LIB] + sources()
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + r.stdout + r.stderr)
    if verbose:
        print(r.stderr)
    build_binding()
    return LIB


def build_binding() -> str:
    cmd = [os.environ.get("CC", "gcc"), "-O2", "-shared", "-fPIC", "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(ROOT, "include"),
           "-o", BINDING, os.path.join(HERE, "csrc", "py_frx.c"), "-L" + HERE, "-l:libfrx.so", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("the Python binding does not compile:\n" + r.stdout + r.stderr)
    return BINDING


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
