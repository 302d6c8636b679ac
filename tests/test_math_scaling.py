"""sw2d_scale_down, the division by a spacing that is a power of two (up to
2^30) where the quotient is subnormal: bit for bit the IEEE product by 2^-k."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "sw2d_math.h"
void down(const double* x, int k, double* y, long n) { for (long i = 0; i < n; i++) y[i] = sw2d_scale_down(x[i], k); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sc")
    (d / "m.c").write_text(SRC)
    subprocess.check_call(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "sw2d_efdc_gb300", "csrc"), str(d / "m.c"), "-o", str(d / "m.so"), "-lm"])
    L = ctypes.CDLL(str(d / "m.so"))
    dp = ctypes.POINTER(ctypes.c_double)
    L.down.argtypes = [dp, ctypes.c_int, dp, ctypes.c_long]
    return L, dp


@pytest.mark.parametrize("k", [1, 2, 11, 12, 13, 14, 20, 30])
def test_subnormal_quotients(lib, k):
    L, dp = lib
    rng = np.random.default_rng(k)
    bits = rng.integers(0, (k + 4) << 52, 200_000, dtype=np.uint64)  # zero to just above the smallest normal times 2^k
    bits[:4] = [0, 1, 1 << 52, ((k + 1) << 52) - 1]
    low = rng.random(bits.size) < 0.3   # halfway cases
    bits[low] &= ~np.uint64((1 << (k - 1)) - 1)
    bits |= rng.integers(0, 2, bits.size, dtype=np.uint64) << np.uint64(63)
    x = bits.view(np.float64)
    y = np.empty_like(x)
    L.down(x.ctypes.data_as(dp), k, y.ctypes.data_as(dp), x.size)
    assert np.array_equal(y.view(np.uint64), (x * 2.0 ** -k).view(np.uint64))
