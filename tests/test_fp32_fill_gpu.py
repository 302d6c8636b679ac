"""FP32 work items cut to fill the GPU: a raster's results do not depend on
whether the engine cuts it into short items (its own choice for rasters that
would leave the GPU idle) or into items of a set length, at sizes around the
ends of strips (224 columns), datum bands (64 rows) and the shortest items,
alone and with every term that has a kernel variant of its own.  Tolerance:
bit-identical; ledger sums are binary32 sums over an item's rows (at most
512), so two splits agree to 512 * 2^-24."""
import numpy as np
import pytest

from oracle import oracle as O
from sw2d_efdc_gb300 import api
from tests.helpers import bumpy_case, model_from_case

pytestmark = pytest.mark.gpu

SIZES = [(25, 20), (64, 224), (65, 225), (130, 448), (203, 449), (515, 230), (1030, 1010)]


@pytest.mark.parametrize("R,C", SIZES)
@pytest.mark.parametrize("terms", [False, True])
def test_short_items_give_the_same_bits(R, C, terms, monkeypatch):
    rng = np.random.default_rng(R + 7 * C)
    kw = dict(frac_int=0.1, frac_lwl=0.02, evap=np.array([0.3, 0.2]), src_cell=np.array([R * C // 2 + 3], np.int32),
              src_q=np.array([[0.5], [0.4]]), dtoq=3600.0) if terms else {}
    case = bumpy_case(R=R, C=C, seed=R, cellsize=5.0, t_end=1e9, dt_mode=O.DT_CFL, cfl=0.7, dt_max=2.0,
                      outflow_south=True, **kw)
    if terms:
        case.rain_weight = rng.random((R, C)).astype(np.float32)
        case.manning_field = rng.choice([0.02, 0.05, 0.10], size=(R, C))

    def run():
        m = model_from_case(case, precision=api.FP32)
        m.step(21)
        m.step(20)
        out = (*m.state(), m.time(), m.ledger())
        m.close()
        return out

    own = run()
    for rows in ("16", "512"):
        monkeypatch.setenv("SW2D_SEGMENT_ROWS", rows)
        fixed = run()
        for a, b in zip(own[:3], fixed[:3]):
            assert np.array_equal(a, b)
        assert own[3] == fixed[3]
        for k in ("rain_in", "source_in", "evap_out", "outflow"):
            assert abs(own[4][k] - fixed[4][k]) <= 512 * 2.0 ** -24 * abs(fixed[4][k]), k
