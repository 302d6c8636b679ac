"""CFL speed of states with depths that are infinite, NaN or negative, and with
thresholds below the binary32 range, in the FP64 step and in the no-allocation
measure.  The speed is the maximum over faces between two active cells whose
mean depth is >= th, in binary64; a face whose mean depth is NaN has none.
Tolerance: bit-identical to numpy's binary64 evaluation of that rule (|q| / hm,
the square root and the sum are single IEEE operations on both sides)."""
import numpy as np
import pytest

from sw2d_efdc_gb300 import api

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

G, ND = 9.80, -9999.0


def _speed(h, qx, qy, dx, th):
    """The rule above; a NaN speed (of a NaN discharge) counts."""
    s = 0.0
    with np.errstate(all="ignore"):
        for a, b, q in ((h[:-1], h[1:], qx[1:-1]), (h[:, :-1], h[:, 1:], qy[:, 1:-1])):
            hm = 0.5 * (a + b)
            v = (np.abs(np.where(q == 0, 0.0, q / hm)) + np.sqrt(G * hm)) * (1.0 / dx)
            v = v[hm >= th]
            s += np.max(v) if v.size else 0.0
    return s


def _stepped(h, dx, th):
    """The step's own speed of the entering state h (discharges zero), as its ledger has it."""
    R, C = h.shape
    m = api.Model(api.default_config(rows=R, cols=C, dx=dx, dy=dx, dt_mode=api.DT_CFL, series_mode=api.SERIES_STEP,
                                     manning=0.03, cfl=0.1, dt_max=0.01, th=th, g=G, nodata=ND))
    m.set_dem(np.zeros((R, C)))
    m.set_rain_series(np.zeros(4), 3600.0)
    m.set_depth(h)
    m.step(1)
    s = m.ledger()["s_max"]
    m.close()
    return s


def _measured(h, dx, th, qx=None, qy=None):
    R, C = h.shape
    qx = np.zeros((R + 1, C)) if qx is None else qx
    qy = np.zeros((R, C + 1)) if qy is None else qy
    a = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (np.zeros((R, C)), h, qx, qy)]
    torch.cuda.synchronize()
    return api.measure_state_noalloc(*[x.data_ptr() for x in a], R, C, dx, dx, ND, th, G)[1]


def _zero_q(h):
    R, C = h.shape
    return np.zeros((R + 1, C)), np.zeros((R, C + 1))


def _nan_beside_deep_water():
    h = np.full((40, 70), 0.01)
    h[10, 20] = 2.0     # the fastest faces, in the same rows of 32 cells as the NaN's
    h[10, 5] = np.nan
    return h


def test_step_nan_hides_no_other_face():
    h = _nan_beside_deep_water()
    got, want = _stepped(h, 10.0, 1e-4), _speed(h, *_zero_q(h), 10.0, 1e-4)
    assert got == want


def test_measure_nan_depth_has_no_speed():
    h = _nan_beside_deep_water()
    got, want = _measured(h, 10.0, 1e-4), _speed(h, *_zero_q(h), 10.0, 1e-4)
    assert got == want


def test_measure_nan_discharge_shows_in_the_speed():
    h = np.full((40, 70), 0.5)
    qx, qy = _zero_q(h)
    qx[7, 9] = np.nan
    assert np.isnan(_measured(h, 10.0, 1e-4, qx, qy))
    qx[7, 9] = np.inf
    assert _measured(h, 10.0, 1e-4, qx, qy) == np.inf


def test_measure_infinite_depth():
    h = np.full((40, 70), 0.5)
    h[3, 4] = np.inf
    assert _measured(h, 10.0, 1e-4) == np.inf


def _cancelling(rng, th, off):
    """Cells of 1 to 1000 m, each beside one negative cell that leaves a mean
    depth of th + off; every other mean is negative."""
    h = np.full((34, 66), -4000.0)
    for r in range(2, 32, 4):
        for c in range(2, 62, 4):
            a = float(rng.uniform(1.0, 1000.0))
            h[r, c] = a
            h[r, c + 1] = 2.0 * (th + off) - a
    return h


@pytest.mark.parametrize("off", [1e-10, -1e-10, 1e-5, -3e-5])
@pytest.mark.parametrize("run", [_stepped, _measured], ids=["step", "measure"])
def test_depths_of_opposite_sign(run, off):
    h = _cancelling(np.random.default_rng(7), 1e-4, off)
    got, want = run(h, 10.0, 1e-4), _speed(h, *_zero_q(h), 10.0, 1e-4)
    assert got == want


@pytest.mark.parametrize("run", [_stepped, _measured], ids=["step", "measure"])
def test_the_fastest_face_between_depths_of_opposite_sign(run):
    h = np.full((34, 66), -4000.0)
    h[4, 4], h[4, 5] = 0.5001, 0.5001
    h[4, 12], h[4, 13] = 1000.0 + 4.8e-4, -999.0  # mean 0.50024; truncated to 21 bits 0.5
    got, want = run(h, 10.0, 1e-4), _speed(h, *_zero_q(h), 10.0, 1e-4)
    assert got == want


@pytest.mark.parametrize("th", [1e-40, 3e-39, 1e-310])
@pytest.mark.parametrize("run", [_stepped, _measured], ids=["step", "measure"])
def test_thresholds_below_binary32(run, th):
    h = np.zeros((20, 40))
    h[5, 6] = 2.5 * th     # mean 1.25 th beside a dry cell
    h[9, 30] = 1.5 * th    # mean 0.75 th
    got, want = run(h, 10.0, th), _speed(h, *_zero_q(h), 10.0, th)
    assert got == want
