"""The device lake-edge pass around the length its list of edge cells may have
(9216 cells in shared memory, a sweep over the diagonals beyond), with chains
of edge cells that wait for one another, NODATA beside them, and updated
values that become NODATA.  Tolerance: bit-identical to the host sweep."""
import numpy as np
import pytest

from sw2d_efdc_gb300 import api

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _edges(m):
    i = m[1:-1, 1:-1]
    return int(((i != 1) & ((i != m[:-2, 1:-1]) | (i != m[2:, 1:-1]) | (i != m[1:-1, :-2]) | (i != m[1:-1, 2:]))).sum())


def _check(mask, dem):
    m = torch.from_numpy(np.ascontiguousarray(mask, np.int32)).cuda()
    z = torch.from_numpy(np.ascontiguousarray(dem, np.float64)).cuda()
    torch.cuda.synchronize()
    api.lake_catchment_smooth_device(dem.shape[0], dem.shape[1], m.data_ptr(), z.data_ptr())
    assert z.cpu().numpy().tobytes() == api.lake_catchment_smooth(mask, dem).tobytes()


@pytest.mark.parametrize("edges", [1, 1023, 1025, 9215, 9216, 9217, 14000])
def test_lists_around_their_limit(edges):
    rng = np.random.default_rng(edges)
    R, C = 460, 461
    mask = np.zeros((R, C), np.int32)
    spots = [(r, c) for r in range(2, R - 2, 3) for c in range(2, C - 2, 3)]
    rng.shuffle(spots)
    n = 0
    for r, c in spots:  # a lone lake cell has four edge neighbours; a lone cell of another kind is an edge with them
        left = edges - n
        if left == 0:
            break
        if left >= 5:
            mask[r, c] = 2
            n += 5
        elif left == 4:
            mask[r, c] = 1
            n += 4
        else:  # a lake cell in the corner of the interior touches fewer inner cells
            break
    dem = rng.normal(20.0, 4.0, (R, C))
    dem[rng.random((R, C)) < 0.02] = -9999.0
    while _edges(mask) < edges:  # top up along the border, where a lake cell has one inner neighbour
        c = int(rng.integers(2, C - 2))
        if mask[0, c] == 0 and (mask[1, c - 1:c + 2] == 0).all() and (mask[2, c] == 0):
            mask[0, c] = 1
    assert _edges(mask) == edges
    _check(mask, dem)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_chains_and_updates_that_become_nodata(seed):
    rng = np.random.default_rng(seed)
    R, C = 90, 70
    mask = rng.integers(0, 4, (R, C)).astype(np.int32)  # nearly every cell an edge: chains in both directions
    dem = rng.normal(0.0, 1.0, (R, C))
    dem[rng.random((R, C)) < 0.15] = -9999.0
    dem[rng.random((R, C)) < 0.15] = -9998.0            # means of -9998 and -10000 are -9999
    dem[rng.random((R, C)) < 0.15] = -10000.0
    assert _edges(mask) <= 9216
    _check(mask, dem)
