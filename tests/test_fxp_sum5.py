"""sum<5> and sum6 (fp64int.cuh), which the 3D sweeps call, return the bits of
the additions they stand for: on the CPU and on the GPU, over the operands of
test_fxp.py."""
import ctypes
import os
import subprocess

import pytest

import test_fxp

SRC = os.path.join(test_fxp.ROOT, "tests", "cuda", "fxp_sum5_check.cu")
D, U = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_ulonglong)


def build(gpu):
    lib = os.path.join(test_fxp.BUILD, f"fxp_sum5_check_{'gpu' if gpu else 'cpu'}.so")
    os.makedirs(test_fxp.BUILD, exist_ok=True)
    newest = max(os.path.getmtime(p) for p in (SRC, test_fxp.SRC, os.path.join(test_fxp.CSRC, "fp64int.cuh")))
    if not os.path.exists(lib) or os.path.getmtime(lib) < newest:
        if gpu:
            nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
            cmd = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false", "-shared",
                   "-Xcompiler", "-fPIC", "-I", test_fxp.CSRC, SRC, "-o", lib]
        else:
            cmd = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++",
                   "-DFXP_CPU", "-I", test_fxp.CSRC, SRC, "-o", lib]
        subprocess.run(cmd, check=True)
    L = ctypes.CDLL(lib)
    L.fxp_random5.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong, U, D]
    L.fxp_rows5.argtypes = [D, ctypes.c_int, U, D]
    return L


def run(L, n):
    bad, first = ctypes.c_ulonglong(), (ctypes.c_double * 7)()
    for seed in (1, 20240503):
        assert L.fxp_random5(n, seed, ctypes.byref(bad), first) == 0
        assert bad.value == 0, (bad.value, [x.hex() for x in first])
    r = test_fxp.rows()
    assert L.fxp_rows5(r.ctypes.data_as(D), len(r), ctypes.byref(bad), first) == 0
    assert bad.value == 0, (bad.value, [x.hex() for x in first])


def test_five_term_sums_have_the_additions_bits_on_the_host():
    run(build(False), 4_000_000)


@pytest.mark.gpu
def test_five_term_sums_have_the_additions_bits_on_the_gpu():
    run(build(True), 1 << 28)
