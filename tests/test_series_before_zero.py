"""Forcing of a clock that starts before time 0: the series are never read
before their first entry.  CPU: the entry's index; GPU (three series modes,
both precisions): FP64 bit-identical to the oracle, which uses the same index,
FP32 within 1 mm of it, its usual tolerance."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from sw2d_efdc_gb300 import api
from tests.helpers import bumpy_case, model_from_case

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_index_stays_in_the_series(tmp_path):
    (tmp_path / "m.c").write_text('#include "sw2d_math.h"\n'
                                  "int at(double t, double d, int n) { return sw2d_series_index(t, d, n); }\n")
    subprocess.check_call(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "sw2d_efdc_gb300", "csrc"), str(tmp_path / "m.c"), "-o",
                           str(tmp_path / "m.so"), "-lm"])
    at = ctypes.CDLL(str(tmp_path / "m.so")).at
    at.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.c_int]
    for t, want in ((-1e300, 0), (-5000.0, 0), (-300.0, 0), (-299.0, 0), (-0.0, 0), (299.0, 0), (300.0, 1), (2999.0, 9),
                    (3000.0, 10), (1e300, 10), (float("nan"), 0)):
        assert at(t, 300.0, 10) == want, t


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [O.RAIN_REFERENCE, O.RAIN_LINEAR, O.RAIN_STEP])
@pytest.mark.parametrize("t0,dts", [(-250.0, 300.0), (-5000.0, 300.0), (-1e8, 0.01)])
def test_runs_before_time_zero(mode, t0, dts):
    R, C = 40, 48
    k = 1e-6 * dts if mode == O.RAIN_STEP else 1e-3 * dts / max(abs(t0), dts)  # rates of 1e-6 m/s or so
    case = bumpy_case(R=R, C=C, seed=4, cellsize=5.0, dt=0.05, t0=t0, t_end=t0 + 1e6, rain=k * np.array([1.0, 1.5, 0.7]),
                      dtrain=dts, rain_mode=mode, evap=0.1 * k * np.array([0.5, 0.4, 0.3]), outflow_south=True)
    case.src_cell = np.array([12 * C + 9, 30 * C + 31], np.int32)
    case.src_q = 1e-3 * np.array([[1.0, 0.5], [0.8, 0.6]]) * (dts / max(abs(t0), dts))
    case.dtoq = dts
    o = O.Oracle(case, math=O.MATH_DEVICE)
    o.run(max_iters=40)
    f = o.fields()
    for precision in (api.FP64, api.FP32):
        m = model_from_case(case, precision)
        m.step(40)
        h, qx, qy = m.state()
        if precision == api.FP64:
            assert np.array_equal(h, f["h"]) and np.array_equal(qx, f["qx"]) and np.array_equal(qy, f["qy"])
        else:
            assert np.abs(h - f["h"]).max() <= 1e-3
        m.close()
