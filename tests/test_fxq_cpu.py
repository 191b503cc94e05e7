"""The integer-pipe quotients of the FP64 kernels (fp64int.cuh) return the
bits of the correctly rounded division, whatever the single-precision seed
within its documented error; the GPU's own division is compared in
test_div_gpu.py."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bsam1.2_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "cuda", "fxq_check.cu")


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_integer_quotients_are_correctly_rounded(tmp_path, ulps):
    lib = str(tmp_path / "fxq.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", "-DFXP_CPU",
                    f"-DFXP_SEED_ULPS=({ulps})", "-I", CSRC, SRC, "-o", lib], check=True)
    L = ctypes.CDLL(lib)
    D = ctypes.POINTER(ctypes.c_double)
    L.fxq_random.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong, D]
    L.fxq_rows.argtypes = [D, ctypes.c_int, D]
    L.fxq_random.restype = L.fxq_rows.restype = ctypes.c_ulonglong
    first = (ctypes.c_double * 3)()
    assert L.fxq_random(4_000_000, 7 + ulps, first) == 0, [x.hex() for x in first]
    u = 2.0 ** -52
    vals = [1.0, 1.0 + u, 1.0 + 2 * u, 1.5, 2.0 - u, 2.0 - 2 * u, 2.0, 3.0, 1 / 3, 0.1, 7.0, 2.0 ** -400, 2.0 ** -401,
            2.0 ** 399 * (2 - u), 2.0 ** 400, 0.5, 1.0 - u / 2, 0.0, 5e-324, 2.0 ** -1022, 1.7976931348623157e308,
            np.inf, np.nan]
    vals += [-v for v in vals]
    r = np.ascontiguousarray(np.array(list(itertools.product(vals, repeat=3))))
    assert L.fxq_rows(r.ctypes.data_as(D), len(r), first) == 0, [x.hex() for x in first]
