"""The device lake-edge pass from several threads and streams: a call does not
wait for another call's stream, and calls side by side give each its own
result."""
import threading
import time

import numpy as np
import pytest

from sw2d_efdc_gb300 import api

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _case(seed, R, C):
    rng = np.random.default_rng(seed)
    r, c = np.mgrid[0:R, 0:C]
    mask = (((r / R - 0.5) ** 2 + (c / C - 0.5) ** 2 + 0.02 * rng.standard_normal((R, C))) < 0.08).astype(np.int32)
    dem = rng.normal(20.0, 4.0, (R, C))
    dem[rng.random((R, C)) < 0.02] = -9999.0
    return mask, dem, api.lake_catchment_smooth(mask, dem)


def _on_device(mask, dem):
    return torch.from_numpy(mask).cuda(), torch.from_numpy(dem).cuda()


def test_a_call_does_not_wait_for_another_stream():
    mask, dem, want = _case(1, 120, 90)
    slow, quick = torch.cuda.Stream(), torch.cuda.Stream()
    m0, z0 = _on_device(mask, dem)
    api.lake_catchment_smooth_device(120, 90, m0.data_ptr(), z0.data_ptr(), quick.cuda_stream)  # code loaded
    m1, z1 = _on_device(mask, dem)
    m2, z2 = _on_device(mask, dem)
    torch.cuda.synchronize()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(3_000_000_000)  # about a second and a half of bounded waiting
    t0 = time.perf_counter()
    first = threading.Thread(target=lambda: api.lake_catchment_smooth_device(
        120, 90, m1.data_ptr(), z1.data_ptr(), slow.cuda_stream))
    first.start()
    time.sleep(0.2)  # the first call is under way
    api.lake_catchment_smooth_device(120, 90, m2.data_ptr(), z2.data_ptr(), quick.cuda_stream)
    t_quick = time.perf_counter() - t0
    first.join()
    t_slow = time.perf_counter() - t0
    assert t_slow > 0.8, "the first call's stream was not busy for long enough to tell"
    assert t_quick < 0.6, (t_quick, t_slow)
    assert z1.cpu().numpy().tobytes() == want.tobytes() and z2.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("threads", [2, 24])
def test_calls_side_by_side_keep_their_own_lists(threads):
    cases = [_case(10 + k, 60 + 37 * k, 200 - 5 * k) for k in range(threads)]
    wrong = []

    def work(k):
        mask, dem, want = cases[k]
        s = torch.cuda.Stream()
        for _ in range(5):
            with torch.cuda.stream(s):
                m, z = _on_device(mask, dem)
            s.synchronize()
            api.lake_catchment_smooth_device(*dem.shape, m.data_ptr(), z.data_ptr(), s.cuda_stream)
            if z.cpu().numpy().tobytes() != want.tobytes():
                wrong.append(k)

    th = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not wrong
