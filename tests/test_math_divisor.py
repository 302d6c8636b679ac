"""sw2d_div_by (division by a fixed spacing on the integer pipes) evaluated on
the CPU: bit for bit the IEEE division, for quotients that are exact, one unit
beside exact and generic, and the same as sw2d_div_const outside the normal
range."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "sw2d_math.h"
void divby(const double* a, double d, double* y, long n) {
    sw2d_divisor c = sw2d_divisor_of(d);
    for (long i = 0; i < n; i++) y[i] = sw2d_div_by(a[i], &c);
}
void divc(const double* a, double d, double* y, long n) { for (long i = 0; i < n; i++) y[i] = sw2d_div_const(a[i], d, 1.0 / d); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("dv")
    (d / "m.c").write_text(SRC)
    subprocess.check_call(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "sw2d_efdc_gb300", "csrc"), str(d / "m.c"), "-o", str(d / "m.so"), "-lm"])
    L = ctypes.CDLL(str(d / "m.so"))
    dp = ctypes.POINTER(ctypes.c_double)
    L.divby.argtypes = L.divc.argtypes = [dp, ctypes.c_double, dp, ctypes.c_long]
    return L, dp


@pytest.mark.parametrize("d", [10.0, 3.0, 1.0, 2.0, 0.5, 0.1, 1.0 / 3.0, 12.34567, 1e-3, 99.99999, 1e300, 4e-308])
def test_division_by_a_spacing_is_the_ieee_division(lib, d):
    L, dp = lib
    rng = np.random.default_rng(4)
    n = 400_000
    a = rng.standard_normal(n) * 10.0 ** rng.uniform(-30, 30, n)
    a[: n // 4] = d * rng.integers(-1 << 20, 1 << 20, n // 4)                       # exact quotients
    a[n // 4: n // 2] = (a[: n // 4].view(np.int64) + rng.integers(-2, 3, n // 4)).view(np.float64)  # beside them
    a = np.ascontiguousarray(a[np.isfinite(a)])
    y, ref = np.empty_like(a), a / d
    L.divby(a.ctypes.data_as(dp), d, y.ctypes.data_as(dp), a.size)
    tiny = 2.3e-308
    ok = (np.abs(a) > tiny) & (np.abs(ref) > tiny) & np.isfinite(ref)
    assert (y[ok].view(np.uint64) == ref[ok].view(np.uint64)).all()
    c = np.empty_like(a)
    L.divc(a.ctypes.data_as(dp), d, c.ctypes.data_as(dp), a.size)
    same = (y.view(np.uint64) == c.view(np.uint64)) | (np.isnan(y) & np.isnan(c))
    assert same[~ok].all()
