"""The FP64 step on both sides of every raster size at which its kernels are
cut differently ((rows + 1)(cols + 1) = 100,000, 300,000, 320,000, 700,000 and
2,000,000) and above the largest, with the last row first and last in a row
of tiles, plain and with the terms whose sums go tile by tile.  Bit-identical
to the oracle's device-math flavour (as every FP64 case); ledger sums, which
are added in another order, within 1e-12."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import bumpy_case, model_from_case

pytestmark = pytest.mark.gpu

# below and at each limit; then 16-row tiles with the last row first (1344 = 84 x 16) and last in its tile
SIZES = [(248, 400), (249, 399), (498, 600), (499, 599), (498, 640), (499, 639), (698, 1000), (699, 999), (1248, 1600),
         (1249, 1599), (1345, 1500), (1344, 1499)]


@pytest.mark.parametrize("R,C", SIZES)
@pytest.mark.parametrize("terms", ["plain", "lake", "field"])
def test_both_sides_of_every_limit(R, C, terms):
    rng = np.random.default_rng(R * 1009 + C)
    kw = {}
    if terms != "plain":
        kw = dict(frac_int=0.1, frac_inf=0.05, frac_lwl=0.02)
    if terms == "lake":
        kw.update(evap=np.array([0.3, 0.2, 0.1]))
    case = bumpy_case(R=R, C=C, seed=R + C, cellsize=3.0, dt=0.02, t_end=1e9, dt_mode=O.DT_CFL, cfl=0.7, dt_max=2.0,
                      outflow_south=True, **kw)
    act = case.dem != -9999.0
    case.h0 = np.where(act & (rng.random((R, C)) < 0.6), case.h0 + 0.1 * rng.random((R, C)), case.h0)
    if terms == "field":
        case.rain_weight = rng.random((R, C)).astype(np.float32)
        case.src_cell = np.array([R * C // 2, (R - 2) * C + C // 2], np.int32)
        case.src_q = np.array([[0.4, 0.2], [0.3, 0.1]])
        case.dtoq = 3600.0
    m = model_from_case(case)
    m.step(5)
    o = O.Oracle(case, math=O.MATH_DEVICE)
    o.run(max_iters=5)
    h, qx, qy = m.state()
    f = o.fields()
    assert m.time()[1] == 5
    assert np.array_equal(h, f["h"]) and np.array_equal(qx, f["qx"]) and np.array_equal(qy, f["qy"])
    led, ref = m.ledger(), o.ledger()
    for k in ("volume", "rain_in", "evap_out", "source_in", "outflow"):
        assert abs(led[k] - ref[k]) <= 1e-12 * max(abs(ref[k]), 1e-300), (k, led[k], ref[k])
    m.close()
