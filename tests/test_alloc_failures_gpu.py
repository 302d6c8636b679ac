"""Failed allocations and launches, made by fakes of the failing calls (the
library's own objects linked with them wrapped): without pinned staging a
raster's inputs go through pageable memory, a scenario or a raster that finds
no device memory does not spoil the ones that run, and after a launch that was
refused state and ledger are those of the iterations that ran.  Results: the
same bits as without the failure."""
import glob
import os
import subprocess
import sys

import numpy as np
import pytest

from sw2d_efdc_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKES = r"""
#include <cuda_runtime.h>
extern "C" {
int fail_pinned = 0, fail_device = 0; /* how many calls to refuse, of cudaMalloc those of 800 kB and more */
int graphs_left = -1;                 /* graph launches until all are refused (-1: never) */
cudaError_t __real_cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t s);
cudaError_t __wrap_cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t s) {
    if (graphs_left == 0) return cudaErrorMemoryAllocation;
    if (graphs_left > 0) graphs_left--;
    return __real_cudaGraphLaunch(g, s);
}
cudaError_t __real_cudaMalloc(void** p, size_t n);
cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
    if (fail_device <= 0 || n < 800000) return __real_cudaMalloc(p, n);
    fail_device--;
    return __real_cudaMalloc(p, (size_t)1 << 60); /* refused by the runtime, which keeps it as its last error, too */
}
cudaError_t __real_cudaMallocHost(void** p, size_t n);
cudaError_t __wrap_cudaMallocHost(void** p, size_t n) {
    if (fail_pinned <= 0) return __real_cudaMallocHost(p, n);
    fail_pinned--;
    void* q = nullptr;
    return __real_cudaMalloc(&q, (size_t)1 << 60);
}
}
"""

RASTER = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from sw2d_efdc_gb300 import api
lib = api.load(sys.argv[2])
R, C = 210, 190
dem = 0.01 * np.arange(R)[::-1, None] + 0.02 * np.random.default_rng(5).standard_normal((R, C))
m = api.Model(api.default_config(rows=R, cols=C, precision=api.FP32, dx=2.0, dy=2.0, dt_mode=api.DT_CFL,
                                 series_mode=api.SERIES_STEP, outflow=api.OUTFLOW_SOUTH, manning=0.03))
m.set_dem(dem)
m.set_rain_series(np.full(4, 5.0), 300.0)
n = ctypes.c_int.in_dll(lib, "fail_pinned")
n.value = int(sys.argv[3])
m.set_depth(np.full((R, C), 0.02))
assert n.value == 0
m.step(20)
np.savez(sys.argv[4], **dict(zip(("h", "qx", "qy"), m.state())))
"""
BATCH = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from sw2d_efdc_gb300 import api
lib = api.load(sys.argv[2])
rng = np.random.default_rng(5)
b = api.Batch()
ids = []
def submit(side):
    dem = 0.01 * np.arange(side)[::-1, None] + 0.02 * rng.standard_normal((side, side))
    ids.append(b.submit(dem=dem, depth=np.full((side, side), 0.02), rain_mm=np.full(4, 5.0), dtrain=300.0, dx=2.0,
                        t_end=20.0, outflow=api.OUTFLOW_SOUTH, manning=0.03))
submit(210)
assert b.step(4) == (1, 0)
submit(230)
n = ctypes.c_int.in_dll(lib, "fail_device")
n.value = int(sys.argv[3])
steps = [b.step(2)]
assert n.value == 0
while steps[-1] != (0, 0):
    steps.append(b.step(16))
out = {"first": np.array(steps[0])}
for k, i in enumerate(ids):
    out["status%d" % k] = np.array(b.poll(i, ledger=False)[0])
    for f, v in zip(("h", "qx", "qy"), b.result(i)):
        out["%s%d" % (f, k)] = v
np.savez(sys.argv[4], **out)
"""

CREATE = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from sw2d_efdc_gb300 import api
lib = api.load(sys.argv[2])
def config(side):
    return api.default_config(rows=side, cols=side, dx=2.0, dy=2.0, dt_mode=api.DT_CFL, series_mode=api.SERIES_STEP,
                              outflow=api.OUTFLOW_SOUTH, manning=0.03)
m = api.Model(config(100))
m.set_dem(0.01 * np.arange(100)[::-1, None] + np.zeros((100, 100)))
m.set_rain_series(np.full(4, 5.0), 300.0)
m.set_depth(np.full((100, 100), 0.02))
n = ctypes.c_int.in_dll(lib, "fail_device")
n.value = int(sys.argv[3])
refused = False
try:
    api.Model(config(1000))
except api.Sw2dError as e:
    refused = e.code == -3
assert refused == bool(int(sys.argv[3])) and n.value == 0
m.step(20)
np.savez(sys.argv[4], **dict(zip(("h", "qx", "qy"), m.state())))
"""

LAUNCH = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from sw2d_efdc_gb300 import api
lib = api.load(sys.argv[2])
m = api.Model(api.default_config(rows=100, cols=90, dx=2.0, dy=2.0, dt_mode=api.DT_CFL, series_mode=api.SERIES_STEP,
                                 outflow=api.OUTFLOW_SOUTH, manning=0.03))
m.set_dem(0.01 * np.arange(100)[::-1, None] + np.zeros((100, 90)))
m.set_rain_series(np.full(4, 5.0), 300.0)
m.set_depth(np.full((100, 90), 0.02))
n = ctypes.c_int.in_dll(lib, "graphs_left")
if int(sys.argv[3]):
    n.value = 2
    try:
        m.step(160)
        assert False
    except api.Sw2dError as e:
        assert e.code == -3
    n.value = -1
else:
    m.step(64)
led = m.ledger()
out = dict(zip(("h", "qx", "qy"), m.state()), ledger=np.array([led[k] for k in sorted(led)]))
m.step(64)
led = m.ledger()
out["later"] = np.array([led[k] for k in sorted(led)])
np.savez(sys.argv[4], **out)
"""


@pytest.fixture(scope="module")
def variant(tmp_path_factory):
    d = tmp_path_factory.mktemp("wrap")
    build.build()
    (d / "fakes.cu").write_text(FAKES)
    so = d / "libsw2d_fakes.so"
    subprocess.check_call([build.nvcc()] + build.ARCH + ["-shared", "-Xcompiler", "-fPIC", str(d / "fakes.cu")] +
                          sorted(glob.glob(os.path.join(build.OBJ_DIR, "*.o"))) +
                          ["-Xlinker", "--wrap=cudaMalloc", "-Xlinker", "--wrap=cudaMallocHost",
                           "-Xlinker", "--wrap=cudaGraphLaunch", "-o", str(so)])
    return d, so


def _run(variant, script, name, *args):
    d, so = variant
    (d / "run.py").write_text(script)
    out = d / (name + ".npz")
    r = subprocess.run([sys.executable, str(d / "run.py"), ROOT, str(so), *map(str, args), str(out)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return dict(np.load(out))


def _same(a, b):
    return a.keys() == b.keys() and all(a[k].tobytes() == b[k].tobytes() for k in a)


def test_no_pinned_staging(variant):
    assert _same(_run(variant, RASTER, "pinned", 1), _run(variant, RASTER, "plain", 0))


def test_no_device_memory_waits(variant):
    late, plain = _run(variant, BATCH, "device", 1), _run(variant, BATCH, "plain", 0)
    assert tuple(late.pop("first")) == (1, 1) and tuple(plain.pop("first")) == (2, 0)
    assert _same(late, plain)


def test_a_raster_that_finds_no_device_memory(variant):
    assert _same(_run(variant, CREATE, "refused", 1), _run(variant, CREATE, "plain", 0))


def test_a_refused_launch_leaves_the_iterations_that_ran(variant):
    assert _same(_run(variant, LAUNCH, "refused", 1), _run(variant, LAUNCH, "plain", 0))
