"""The integer-pipe sums of the FP64 kernels (fp64int.cuh) return the bits of
the round-to-nearest additions they stand for: on the CPU, with the header
compiled by the host compiler, and on the GPU."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bsam1.2_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "cuda", "fxp_check.cu")
BUILD = os.path.join(ROOT, "bsam1.2_gb300", "_build")


def build(gpu):
    lib = os.path.join(BUILD, "fxp_check_gpu.so" if gpu else "fxp_check_cpu.so")
    os.makedirs(BUILD, exist_ok=True)
    newest = max(os.path.getmtime(SRC), os.path.getmtime(os.path.join(CSRC, "fp64int.cuh")))
    if not os.path.exists(lib) or os.path.getmtime(lib) < newest:
        if gpu:
            nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
            cmd = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false", "-shared",
                   "-Xcompiler", "-fPIC", "-I", CSRC, SRC, "-o", lib]
        else:
            cmd = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++",
                   "-DFXP_CPU", "-I", CSRC, SRC, "-o", lib]
        subprocess.run(cmd, check=True)
    L = ctypes.CDLL(lib)
    U, D = ctypes.POINTER(ctypes.c_ulonglong), ctypes.POINTER(ctypes.c_double)
    L.fxp_random.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong, U, D]
    L.fxp_rows.argtypes = [D, ctypes.c_int, U, D]
    return L


def rows():
    """Edge cases: every value beside its neighbours, zeros, subnormals, the
    ends of the exponent range, infinities and NaN, ties, sticky bits at the
    frame's edge, full cancellation."""
    u = 2.0 ** -52
    vals = [1.0, -1.0, 1.0 + u, -(1.0 + u), 2.0 - u, 1.5, u, 2.0 ** -6, -2.0 ** -7 * (1 + u), 2.0 ** -53, 2.0 ** -59,
            -2.0 ** -60, 2.0 ** -31 * (1 + 3 * u), -2.0 ** -32, 0.0, -0.0, 5e-324, 2.0 ** -1022, 2.0 ** -890, 1e300,
            -1.7976931348623157e308, np.inf, -np.inf, np.nan, 1 / 3, -0.1]
    out = [list(p) + [p[0], p[1], p[2], p[0]] for p in itertools.product(vals, repeat=3)]
    out += [[a, b, -a, -b, a, b, (a + b) / 6] for a in vals for b in vals]
    return np.ascontiguousarray(np.array(out, dtype=np.float64))


def run(L, n):
    D = ctypes.POINTER(ctypes.c_double)
    bad, first = ctypes.c_ulonglong(), (ctypes.c_double * 7)()
    for seed in (1, 20240503):
        assert L.fxp_random(n, seed, ctypes.byref(bad), first) == 0
        assert bad.value == 0, (bad.value, [x.hex() for x in first])
    r = rows()
    assert L.fxp_rows(r.ctypes.data_as(D), len(r), ctypes.byref(bad), first) == 0
    assert bad.value == 0, (bad.value, [x.hex() for x in first])


def test_integer_sums_have_the_additions_bits_on_the_host():
    run(build(False), 4_000_000)


@pytest.mark.gpu
def test_integer_sums_have_the_additions_bits_on_the_gpu():
    run(build(True), 1 << 28)
