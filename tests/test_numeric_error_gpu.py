"""A run to an end time that meets a NaN discharge at its outlet: the error is
reported, with the iterations that ran and their time."""
import ctypes

import numpy as np
import pytest

from sw2d_efdc_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seconds", [2.0, 40.0])
def test_iterations_of_a_failing_run_are_reported(seconds):
    R, C = 40, 50
    m = api.Model(api.default_config(rows=R, cols=C, dx=10.0, dy=10.0, dt_mode=api.DT_CFL, series_mode=api.SERIES_STEP,
                                     outflow=api.OUTFLOW_SOUTH, manning=0.03, cfl=0.7, dt_max=0.5))
    m.set_dem(np.zeros((R, C)))
    m.set_rain_series(np.zeros(4), 3600.0)
    h = np.full((R, C), 0.01)
    h[R - 1, 7] = np.nan
    m.set_depth(h)
    n = ctypes.c_int64(-1)
    rc = api.load().sw2d_advance(m._h, ctypes.c_double(seconds), ctypes.byref(n))
    assert rc == api.SW2D_ERR_NUMERIC
    t, iters = m.time()
    assert n.value == iters > 0 and t > 0.0 and m.timing()[0] > 0.0
    m.close()
