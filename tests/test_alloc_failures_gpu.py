"""Failed allocations, made by a fake of the failing call (the library's own
objects linked with it wrapped): without pinned staging a raster's inputs go
through pageable memory.  Results: the same bits as without the failure."""
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
int fail_pinned = 0; /* how many calls to refuse */
cudaError_t __real_cudaMallocHost(void** p, size_t n);
cudaError_t __wrap_cudaMallocHost(void** p, size_t n) {
    if (fail_pinned <= 0) return __real_cudaMallocHost(p, n);
    fail_pinned--;
    void* q = nullptr;
    return cudaMalloc(&q, (size_t)1 << 60); /* refused by the runtime, which keeps it as its last error, too */
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

@pytest.fixture(scope="module")
def variant(tmp_path_factory):
    d = tmp_path_factory.mktemp("wrap")
    build.build()
    (d / "fakes.cu").write_text(FAKES)
    so = d / "libsw2d_fakes.so"
    subprocess.check_call([build.nvcc()] + build.ARCH + ["-shared", "-Xcompiler", "-fPIC", str(d / "fakes.cu")] +
                          sorted(glob.glob(os.path.join(build.OBJ_DIR, "*.o"))) +
                          ["-Xlinker", "--wrap=cudaMallocHost", "-o", str(so)])
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
