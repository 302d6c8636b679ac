"""The binary32 estimates that spare the FP64 step its binary64 operations,
evaluated on the CPU: what they decide is what binary64 decides, over depths
and discharges of both signs, cancelling ones, infinities and NaN."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "sw2d_math.h"
void dry(const double* v, double src, double dt2, double dx, double dy, double th, int* out, long n) {
    for (long i = 0; i < n; i++) {
        const double* q = v + 5 * i;
        const float s = sw2d_f32_est_of_f64(src);
        out[i] = sw2d_dry_est(sw2d_f32_est_hi(q[0]), sw2d_f32_est_hi(q[1]), sw2d_f32_est_hi(q[2]), sw2d_f32_est_hi(q[3]),
                              sw2d_f32_est_hi(q[4]), s, fabsf(s), sw2d_f32_est_of_f64(dt2), (float)(1.0 / dx),
                              (float)(1.0 / dy), (float)th);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pf")
    (d / "m.c").write_text(SRC)
    subprocess.check_call(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "sw2d_efdc_gb300", "csrc"), str(d / "m.c"), "-o", str(d / "m.so"), "-lm"])
    L = ctypes.CDLL(str(d / "m.so"))
    dp, db = ctypes.POINTER(ctypes.c_double), ctypes.c_double
    L.dry.argtypes = [dp, db, db, db, db, db, ctypes.POINTER(ctypes.c_int), ctypes.c_long]
    return L


def _dry(lib, v, src, dt2, dx, dy, th):
    v = np.ascontiguousarray(v)
    out = np.empty(len(v), np.int32)
    lib.dry(v.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), src, dt2, dx, dy, th,
            out.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), len(v))
    with np.errstate(all="ignore"):
        hs = v[:, 0] - dt2 * ((v[:, 2] - v[:, 1]) / dx + (v[:, 4] - v[:, 3]) / dy - src)
    return out, hs


@pytest.mark.parametrize("dt2,dx,th,src", [(0.08, 10.0, 1e-4, 0.0), (1.3, 2.0, 1e-4, 3e-6), (0.004, 0.1, 1e-3, -1e-7),
                                           (30.0, 100.0, 0.01, 1e-3)])
def test_dry_decisions_are_binary64s(lib, dt2, dx, th, src):
    rng = np.random.default_rng(int(dx * 10))
    n = 400_000
    v = rng.standard_normal((n, 5)) * 10.0 ** rng.uniform(-6, 4, (n, 1))
    v[:, 1:] *= 10.0 ** rng.uniform(-6, 2, (n, 4))
    near = rng.random(n) < 0.6  # depths that the divergence takes to th, or a little off it
    hs = v[:, 0] - dt2 * ((v[:, 2] - v[:, 1]) / dx + (v[:, 4] - v[:, 3]) / dx - src)
    off = rng.standard_normal(n) * 10.0 ** rng.uniform(-13, -4, n)
    v[near, 0] += (th + off - hs)[near]
    out, hs = _dry(lib, v, src, dt2, dx, dx, th)
    known = out != 2
    # what binary64's own rounding of hs leaves open is not the estimate's to decide
    mag = np.abs(v[:, 0]) + dt2 * np.abs(v[:, 1:]).sum(1) / dx
    sure = np.abs(hs - th) > 1e-14 * mag
    assert (known & sure).any() and (~known).any()
    assert ((out == 1) == (hs < th))[known & sure].all()


def test_infinities_and_nan_are_left_to_binary64(lib):
    rng = np.random.default_rng(2)
    for bad in (np.inf, -np.inf, np.nan, 1e39, -1e300):
        for k in range(5):
            v = rng.random((64, 5))
            v[:, k] = bad
            out, _ = _dry(lib, v, 0.0, 1e-3, 100.0, 100.0, 1e-4)
            assert (out == 2).all(), (bad, k)
