"""Builds and loads tests/harness/kernel_harness.cu: single kernels of libpibem_gb300.so for the
tests that need more than the C ABI shows (GPU tests only)."""
import ctypes as C
import functools
import os
import subprocess
import tempfile

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "pi-bem_gb300")


@functools.lru_cache(maxsize=None)
def load():
    out = os.path.join(tempfile.mkdtemp(prefix="kernel_harness_"), "libkh.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", "-o", out, os.path.join(REPO, "tests", "harness", "kernel_harness.cu"),
                    "-L" + PKG, "-l:libpibem_gb300.so", "-Xlinker", "-rpath," + PKG], check=True)
    return C.CDLL(out)


def ptr(a, t):
    """The data of a C-contiguous array as a pointer to t."""
    assert a.flags.c_contiguous
    return a.ctypes.data_as(C.POINTER(t))
