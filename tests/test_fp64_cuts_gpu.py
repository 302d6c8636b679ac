"""The FP64 step at the sizes where its kernels are cut differently: one cell
around the edges of the flux blocks (32 x 2, 32 x 8) and of the update tiles
(32 x 4, 32 x 8, 64 x 16), and around the raster sizes at which the cut
changes.  Bit-identical to the oracle's device-math flavour (as every FP64
case); ledger sums, which are added in another order, within 1e-12."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import bumpy_case, model_from_case

pytestmark = pytest.mark.gpu

# (rows, cols): 32 x 4 tiles below 38,912 faces' cells, 32 x 8 below 622,592, then 64 x 16
SIZES = [(31, 63), (32, 64), (33, 31), (197, 196), (198, 196), (278, 279), (280, 278), (255, 319), (788, 788),
         (790, 789), (640, 1023)]


@pytest.mark.parametrize("R,C", SIZES)
@pytest.mark.parametrize("cell", [10.0, 2.0])
def test_every_cut_is_bitwise_the_oracle(R, C, cell):
    rng = np.random.default_rng(R * 1009 + C)
    lake = cell == 10.0
    case = bumpy_case(R=R, C=C, seed=R + C, cellsize=cell, dt=0.02, t_end=1e9, dt_mode=O.DT_CFL, cfl=0.7, dt_max=2.0,
                      outflow_south=True, frac_int=0.1 if lake else 0.0, frac_lwl=0.02 if lake else 0.0,
                      evap=np.array([0.3, 0.2, 0.1]) if lake else None)
    film = rng.random((R, C)) < 0.6
    case.h0 = np.where(film & (case.dem != -9999.0), case.h0 + 0.02 * rng.random((R, C)), case.h0)
    if not lake:
        case.rain_weight = rng.random((R, C)).astype(np.float32)
        case.manning_field = rng.choice([0.02, 0.05, 0.10], size=(R, C))
    m = model_from_case(case)
    m.step(10)
    m.step(3)
    o = O.Oracle(case, math=O.MATH_DEVICE)
    o.run(max_iters=13)
    h, qx, qy = m.state()
    f = o.fields()
    assert m.time()[1] == 13
    assert np.array_equal(h, f["h"]) and np.array_equal(qx, f["qx"]) and np.array_equal(qy, f["qy"])
    led, ref = m.ledger(), o.ledger()
    for k in ("volume", "rain_in", "evap_out", "outflow"):
        assert abs(led[k] - ref[k]) <= 1e-12 * max(abs(ref[k]), 1e-300), (k, led[k], ref[k])
    m.close()
