"""The workloads this library's speed is judged by.

Each case is work that a user's program asks of the library through its Python
mirror (sw2d_efdc_gb300.api, itself a thin layer over the C ABI): a raster
that is already set up is advanced to the next output and its fields are read,
scenarios are served from a queue, a caller's own device state is measured, a
coupled run's DEM is smoothed.  Inputs are synthetic and follow the shapes of
the workloads the repository names (256 x 256 plain run, 701 x 556 coupled
lake, 4096 x 4096 pond break, 8192 x 8192 precision raster, scenarios from 128
cells a side), with thin films, ponds, dry ground and NODATA in them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sw2d_efdc_gb300 import api

NODATA = -9999.0
TH, G = 1e-4, 9.80
EV_WL_MIN = 0.05
MANNING = 0.03

# Defaults of a raster case; a case states only where it differs.
RASTER = {
    "kind": "raster", "precision": "fp64", "rows": 256, "cols": 256, "dx": 10.0, "iters": 32,
    "dt_mode": "cfl",       # "fixed": the reference's own loop with this dt
    "dt": 0.04,
    "advance": False,       # advance(t + seconds) instead of step(iters)
    "seconds": 0.0,
    "series": "step",       # "reference" | "linear" | "step"
    "terrain": "plane",     # "fractal": 40 m of relief with a carved channel
    "classes": 0,           # Manning classes in the raster (0: one uniform n)
    "rain_field": False, "lake": False, "sources": 0, "outflow": False, "holes": False, "reservoir": False,
    "couple": False,        # a lake mask: boundary discharges and velocities are read too
    "read": "state",        # "depth": the depth alone is read
}


def _raster(**kw):
    return {**RASTER, **kw}


def listed():
    return [
        # a very small raster run for a few steps of the reference's loop, as in a calibration sweep or a unit
        # of a larger program: latency and launches
        _raster(name="fp64_33x41", rows=33, cols=41, dx=5.0, iters=10, advance=True, seconds=0.8, dt_mode="fixed",
                series="reference", holes=True),
        # the 256 x 256 plain run from one minute of output to the next: CFL steps, free south outlet
        _raster(name="fp64_256", rows=256, cols=256, dx=10.0, iters=54, advance=True, seconds=60.0, outflow=True),
        # the coupled lake's raster with all its terms: fixed dt, evaporation and loss fractions, a point
        # source, boundary discharges for the lake model at each output
        _raster(name="fp64_701x556_coupled", rows=701, cols=556, dx=10.0, iters=50, advance=True, seconds=4.0,
                dt_mode="fixed", series="reference", lake=True, sources=1, holes=True, couple=True),
        # an irregular catchment: odd sizes, a spacing that is no power of two, many roughness classes
        _raster(name="fp64_1531x1207", rows=1531, cols=1207, dx=3.0, iters=16, series="linear", classes=40,
                holes=True, outflow=True),
        # the headline plain run: pond break on fractal terrain with land cover and a rain field
        _raster(name="fp64_4096_pondbreak", rows=4096, cols=4096, dx=2.0, iters=32, terrain="fractal", classes=3,
                rain_field=True, reservoir=True),
        # the precision form on a small raster: one forecast window of a small catchment
        _raster(name="fp32_200x310", precision="fp32", rows=200, cols=310, dx=5.0, iters=64, outflow=True),
        # the precision form with every term that has a variant of its own
        _raster(name="fp32_1537x1001_terms", precision="fp32", rows=1537, cols=1001, dx=2.0, iters=64,
                terrain="fractal", classes=3, rain_field=True, lake=True, sources=5, holes=True),
        # the precision form's ordinary size
        _raster(name="fp32_2048", precision="fp32", rows=2048, cols=2048, dx=1.0, iters=64, outflow=True),
        # the precision form's largest raster; the depth map is what is read
        _raster(name="fp32_8192", precision="fp32", rows=8192, cols=8192, dx=1.0, iters=96, outflow=True,
                read="depth"),
        # scenarios of uneven size served together from submission to results
        {"name": "batch_16", "kind": "batch", "scenarios": 16, "lo": 128, "hi": 768, "seconds": 60.0, "chunk": 64,
         "classes": 3},
        # volume and CFL speed of a state that another program holds on the device
        {"name": "measure_4096x3000", "kind": "measure", "rows": 4096, "cols": 3000, "dx": 2.0},
        # the lake-edge pre-pass of a coupled run on a DEM that is already on the device
        {"name": "lake_smooth_701x556", "kind": "lake", "rows": 701, "cols": 556},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "fp64", "fp32", "fp32", "fp32", "batch", "measure", "lake"])
    if kind == "batch":
        return {"kind": "batch", "scenarios": rng.randint(2, 16), "lo": _log(rng, 48, 160), "hi": _log(rng, 200, 760),
                "seconds": rng.uniform(20.0, 60.0), "chunk": rng.choice([16, 32, 64]), "classes": rng.choice([0, 3])}
    if kind == "measure":
        return {"kind": "measure", "rows": _log(rng, 30, 4096), "cols": _log(rng, 30, 4096),
                "dx": rng.choice([1.0, 2.0, 3.0, 10.0])}
    if kind == "lake":
        return {"kind": "lake", "rows": _log(rng, 40, 2048), "cols": _log(rng, 40, 1536)}
    rows, cols = _log(rng, 24, 3000), _log(rng, 24, 3000)
    cells = rows * cols
    fixed = rng.random() < 0.3
    terrain = rng.choice(["plane", "plane", "fractal"])
    c = _raster(precision=kind, rows=rows, cols=cols, dx=rng.choice([1.0, 2.0, 3.0, 5.0, 10.0]),
                iters=max(8, min(64, int(1.5e8 / cells))), terrain=terrain,
                classes=rng.choice([0, 0, 3, 40]), rain_field=rng.random() < 0.4, lake=rng.random() < 0.3,
                sources=rng.choice([0, 0, 1, 5]), outflow=rng.random() < 0.5, holes=rng.random() < 0.5)
    if fixed:
        c["dt_mode"], c["dt"] = "fixed", 0.01 if c["dx"] < 3.0 else 0.04
        c["series"] = rng.choice(["reference", "linear", "step"])
        c["advance"], c["seconds"] = True, c["iters"] * 2 * c["dt"]
    else:
        c["series"] = rng.choice(["linear", "step"])
    return c


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _field(rows, cols, dx, amp, g):
    """Stationary random field of unit standard deviation with the spectrum amp(|k|)."""
    dev = _device()
    ky = torch.fft.fftfreq(rows, d=dx, device=dev)[:, None]
    kx = torch.fft.rfftfreq(cols, d=dx, device=dev)[None, :]
    noise = torch.randn(rows, cols, generator=g, device=dev)
    f = torch.fft.irfft2(torch.fft.rfft2(noise) * amp(torch.sqrt(kx * kx + ky * ky)), s=(rows, cols))
    f = f - f.mean()
    return (f / f.std().clamp_min(1e-20)).double()


def _smooth_amp(corr):
    return lambda k: torch.exp(-((2.0 * math.pi * k * corr) ** 2) / 8.0)


def _fractal_amp(hurst):
    return lambda k: torch.where(k > 0, k.clamp_min(1e-12) ** (-(hurst + 1.0)), torch.zeros_like(k))


def _terrain(c, g):
    """DEM and wet initial depth: a film on all slopes, ponds in hollows, some dry ground."""
    rows, cols, dx = c["rows"], c["cols"], c["dx"]
    dev = _device()
    r = torch.arange(rows, device=dev, dtype=torch.float64)[:, None]
    cc = torch.arange(cols, device=dev, dtype=torch.float64)[None, :]
    if c["terrain"] == "fractal":
        f = _field(rows, cols, dx, _fractal_amp(0.8), g)
        relief = min(40.0, 0.005 * min(rows, cols) * dx)
        z = (f - f.min()) * (relief / (f.max() - f.min()).clamp_min(1e-12))
        centre = cols / 2 + 0.15 * cols * torch.sin(2 * math.pi * r / (0.8 * rows))
        channel = (1.0 - (cc - centre).abs() / max(cols // 400, 3)).clamp(0.0, 1.0)
        z = z - min(4.0, 0.2 * relief) * channel
        pond = 0.3 * channel
    else:
        bumps = 0.3 * _field(rows, cols, dx, _smooth_amp(50.0), g)
        z = 0.01 * dx * (rows - 0.5 - r) + bumps
        pond = (-(bumps + 0.4)).clamp_min(0.0)
    film = 0.006 * torch.exp(0.5 * _field(rows, cols, dx, _smooth_amp(20.0 * dx), g))
    dry = _field(rows, cols, dx, _smooth_amp(12.0 * dx), g) > 1.5
    h = torch.where(dry, torch.zeros_like(film), film) + pond
    if c["reservoir"]:
        s = max(4, min(rows, cols) // 10)
        h[rows // 4:rows // 4 + s, cols // 4:cols // 4 + s] = 5.0
    if c["holes"]:
        # a catchment outline and inner gaps without data
        out = ((r / rows - 0.5) ** 2 + (cc / cols - 0.5) ** 2) > 0.40
        gap = _field(rows, cols, dx, _smooth_amp(15.0 * dx), g) > 2.3
        z = torch.where(out | gap, torch.full_like(z, NODATA), z)
        h = torch.where(out | gap, torch.zeros_like(h), h)
    return z, h


def _classes(c, g):
    """Land-cover patches: the class raster and its table of n."""
    k = c["classes"]
    f = _field(c["rows"], c["cols"], c["dx"], _smooth_amp(30.0 * c["dx"]), g)
    u = 0.5 * (1.0 + torch.erf(f / math.sqrt(2.0)))
    cls = (u * k).long().clamp(0, k - 1).to(torch.uint8)
    return cls, np.array([0.02, 0.05, 0.10]) if k == 3 else np.linspace(0.02, 0.12, k)


def _inputs(c, seed):
    """Every input of a raster case, on the torch device (series on the host)."""
    g = _gen(seed)
    rng = np.random.default_rng(seed)
    d = {}
    d["z"], d["h"] = _terrain(c, g)
    d["cls"], d["table"] = _classes(c, g) if c["classes"] else (None, None)
    d["weight"] = None
    if c["rain_field"]:
        w = torch.exp(0.5 * _field(c["rows"], c["cols"], c["dx"], _smooth_amp(200.0), g))
        d["weight"] = (w / w.mean()).float()
    d["rain"] = rng.gamma(0.8, 20.0 / 0.8, 4096) * 300.0 / 3600.0 + 0.2   # mm per 5 minutes
    d["dtrain"] = 300.0
    d["evap"] = 0.02 + 0.02 * rng.random(4096) if c["lake"] else None
    d["src"] = d["srcq"] = None
    if c["sources"]:
        n = c["rows"] * c["cols"]
        inside = np.flatnonzero((d["z"] != NODATA).cpu().numpy().reshape(-1))
        d["src"] = rng.choice(inside if len(inside) >= c["sources"] else n, c["sources"], replace=False).astype(np.int32)
        d["srcq"] = 0.2 + 0.3 * rng.random((512, c["sources"]))
    d["frac"] = (0.10, 0.05, 0.02) if c["lake"] else (0.0, 0.0, 0.0)   # interception, infiltration, lake loss
    return d


def _lake_mask(rows, cols):
    """Lake (1) and catchment (0) cells of a coupled run: part of its geometry, not of its seed."""
    dev, g = _device(), _gen(rows * 4099 + cols)
    r = torch.arange(rows, device=dev, dtype=torch.float64)[:, None] / rows - 0.55
    cc = torch.arange(cols, device=dev, dtype=torch.float64)[None, :] / cols - 0.45
    ragged = 0.02 * _field(rows, cols, 1.0, _smooth_amp(0.04 * min(rows, cols)), g)
    lake = r * r + cc * cc + ragged < 0.06
    return lake.to(torch.int32)


def _batch_inputs(c, seed):
    sides = np.random.default_rng(c["scenarios"] * 10007 + c["hi"])
    sides = np.exp(sides.uniform(math.log(c["lo"]), math.log(c["hi"]), c["scenarios"])).astype(int)
    out = []
    for k, side in enumerate(sides):
        sub = _raster(rows=int(side), cols=int(side), dx=1.0, terrain="fractal" if k % 2 else "plane",
                      classes=c["classes"])
        d = _inputs(sub, seed * 1009 + k)
        kw = {"dem": d["z"].cpu().numpy(), "depth": d["h"].cpu().numpy(), "rain_mm": d["rain"][:72], "dtrain": 300.0,
              "dx": 1.0, "t_end": float(c["seconds"]), "outflow": api.OUTFLOW_SOUTH, "manning": MANNING}
        if d["cls"] is not None:
            kw["manning_classes"], kw["manning_table"] = d["cls"].cpu().numpy(), d["table"]
        out.append(kw)
    return out


def _measure_inputs(c, seed):
    """A wet state on the device: depth and discharges in the layouts the library reads and writes."""
    full = _raster(rows=c["rows"], cols=c["cols"], dx=c["dx"], terrain="fractal", holes=True)
    g = _gen(seed)
    z, h = _terrain(full, g)
    rows, cols = c["rows"], c["cols"]
    qx = 0.02 * torch.randn(rows + 1, cols, generator=g, device=z.device, dtype=torch.float64)
    qy = 0.02 * torch.randn(rows, cols + 1, generator=g, device=z.device, dtype=torch.float64)
    act = z != NODATA
    wet = act & (h > TH)
    qx[1:-1] *= (wet[1:] & wet[:-1])
    qy[:, 1:-1] *= (wet[:, 1:] & wet[:, :-1])
    qx[0] = qx[-1] = 0.0
    qy[:, 0] = qy[:, -1] = 0.0
    return z, h, qx, qy


# ---------------------------------------------------------------- the calls


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "batch":
        return {"case": c, "batch": api.Batch(), "requests": _batch_inputs(c, seed)}
    if c["kind"] == "measure":
        return {"case": c, "arrays": _measure_inputs(c, seed)}
    if c["kind"] == "lake":
        g = _gen(seed)
        z = _terrain(_raster(rows=c["rows"], cols=c["cols"], holes=True), g)[0]
        mask = _lake_mask(c["rows"], c["cols"])
        return {"case": c, "mask": mask, "dem": z.contiguous()}
    d = _inputs(c, seed)
    fi, ff, fl = d["frac"]
    cfg = api.default_config(
        rows=c["rows"], cols=c["cols"], dx=c["dx"], dy=c["dx"],
        precision=api.FP32 if c["precision"] == "fp32" else api.FP64,
        dt_mode=api.DT_FIXED if c["dt_mode"] == "fixed" else api.DT_CFL,
        series_mode={"reference": api.SERIES_REFERENCE, "linear": api.SERIES_LINEAR, "step": api.SERIES_STEP}[c["series"]],
        outflow=api.OUTFLOW_SOUTH if c["outflow"] else api.OUTFLOW_NONE, manning=MANNING, dt=c["dt"], cfl=0.7,
        dt_max=2.0, th=TH, g=G, nodata=NODATA, frac_int=fi, frac_inf=ff, frac_lwl=fl, ev_wl_min=EV_WL_MIN)
    m = api.Model(cfg)
    m.set_dem(d["z"].cpu().numpy())
    if d["cls"] is not None:
        m.set_manning_classes(d["cls"].cpu().numpy(), d["table"])
    m.set_rain_series(d["rain"], d["dtrain"])
    if d["weight"] is not None:
        m.set_rain_field(d["weight"].cpu().numpy())
    if d["evap"] is not None:
        m.set_evaporation_series(d["evap"])
    if d["src"] is not None:
        m.set_point_sources(d["src"], d["srcq"], 3600.0)
    if c["couple"]:
        m.set_coupling_mask(_lake_mask(c["rows"], c["cols"]).cpu().numpy(), lagged=False)
    m.set_depth(d["h"].cpu().numpy())
    return {"case": c, "model": m}


def _run_batch(st):
    b, c = st["batch"], st["case"]
    ids = [b.submit(**kw) for kw in st["requests"]]
    while b.step(c["chunk"]) != (0, 0):
        pass
    out = []
    for rid in ids:
        out += b.result(rid)
        b.release(rid)
    return out


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        return _run_batch(state)
    if c["kind"] == "measure":
        z, h, qx, qy = state["arrays"]
        return api.measure_state_noalloc(z.data_ptr(), h.data_ptr(), qx.data_ptr(), qy.data_ptr(), c["rows"], c["cols"],
                                         c["dx"], c["dx"], NODATA, TH, G, torch.cuda.current_stream().cuda_stream)
    if c["kind"] == "lake":
        z = state["dem"].clone()
        api.lake_catchment_smooth_device(c["rows"], c["cols"], state["mask"].data_ptr(), z.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
        return z
    m = state["model"]
    if c["advance"]:
        t, _ = m.time()
        m.advance(t + c["seconds"])
    else:
        m.step(c["iters"])
    t, _ = m.time()
    out = {"t": t}
    if c["read"] == "depth":
        out["depth"] = m.depth()
    else:
        out["depth"], out["qx"], out["qy"] = m.state()
    if c["couple"]:
        out["uu"], out["vv"] = m.velocity()
        out["boundary"] = m.couple_sample()
    return out


def work(case):
    c = case
    if c["kind"] == "batch":
        side2 = (c["hi"] ** 2 - c["lo"] ** 2) / (2.0 * math.log(c["hi"] / c["lo"])) if c["hi"] > c["lo"] else c["lo"] ** 2
        n = 20.0 * c["seconds"] * side2 * c["scenarios"]      # about twenty iterations a simulated second at 1 m
        return {"bytes": 38.0 * n, "flops": 150.0 * n}
    cells = c["rows"] * c["cols"]
    if c["kind"] == "measure":
        return {"bytes": 32.0 * cells, "flops": 12.0 * cells}
    if c["kind"] == "lake":
        return {"bytes": 20.0 * cells, "flops": 0.1 * cells}
    # an iteration: depth and both discharges read and written once, the bed, a flag, class and weight read
    per = 56.0 + 1.0 if c["precision"] == "fp64" else 36.0 + 1.0
    per += (1.0 if c["classes"] else 0.0) + (4.0 if c["rain_field"] else 0.0)
    out = 8.0 * cells * (1 if c["read"] == "depth" else 3) + (16.0 * cells if c["couple"] else 0.0)
    return {"bytes": per * cells * c["iters"] + out, "flops": 150.0 * cells * c["iters"]}


# ---------------------------------------------------------------- the step in 64 bits


def _series(v, dts, t, mode):
    n = len(v)
    at = lambda k: float(v[k]) if k < n else 0.0  # noqa: E731
    if mode == "reference" and t <= 1.0:
        return at(0) * t
    it = min(int(t / dts), n)
    if mode == "step":
        return at(it)
    d = at(it + 1) - at(it)
    return at(it) + (d / (dts * (t - dts * it)) if mode == "reference" else d * ((t - dts * it) / dts))


class _Step64:
    """The SW2D iteration in binary64 torch operations: flux of every face, depth at t, outflow of cells that
    would fall dry closed, depth at t + dt."""

    def __init__(self, c, d):
        self.c, self.d = c, d
        self.R, self.C = c["rows"], c["cols"]
        z, h = d["z"], d["h"]
        self.act = z != NODATA
        self.z = z
        self.h = torch.where(self.act, h, torch.zeros_like(h))
        dev = z.device
        # face arrays with two rings around the raster, as are the padded cells below
        self.qx, self.qy, self.u, self.v = (torch.zeros(self.R + 4, self.C + 4, dtype=torch.float64, device=dev)
                                            for _ in range(4))
        n = d["table"] if d["cls"] is not None else np.array([MANNING])
        cls = d["cls"].long() if d["cls"] is not None else torch.zeros_like(z, dtype=torch.long)
        self.n = torch.as_tensor(np.asarray(n), device=dev, dtype=torch.float64)[cls]
        self.w = d["weight"].double() if d["weight"] is not None else None
        self.area = c["dx"] * c["dx"]
        self.t = 0.0
        self.S = self.speed()

    def pad(self, a):
        return torch.nn.functional.pad(a, (2, 2, 2, 2))

    def at(self, a, dr=0, dc=0):
        """Padded array seen from the faces (r, c), r in 0..R, c in 0..C."""
        return a[2 + dr:3 + dr + self.R, 2 + dc:3 + dc + self.C]

    def put(self, a):
        return torch.nn.functional.pad(a, (2, 1, 2, 1))

    def speed(self):
        h, act, dx = self.h, self.act, self.c["dx"]
        s = 0.0
        for dim, vel in ((0, self.u[3:2 + self.R, 2:2 + self.C]), (1, self.v[2:2 + self.R, 3:2 + self.C])):
            m = h.shape[dim] - 1
            hm = 0.5 * (h.narrow(dim, 1, m) + h.narrow(dim, 0, m))
            ok = act.narrow(dim, 1, m) & act.narrow(dim, 0, m) & (hm >= TH)
            s += float(torch.where(ok, (vel.abs() + torch.sqrt(G * hm)) / dx, torch.zeros_like(hm)).max())
        return s

    def special(self, ha, hb, za, zb, act):
        """Kind of each face and the discharge of the weir and dry-bed ones."""
        wa, wb = ha > TH, hb > TH
        ea, eb = ha + za, hb + zb
        open_ = act & (wa | wb)
        k2 = open_ & (eb < za)
        k3 = open_ & ~k2 & (ea < zb)
        k4 = open_ & ~k2 & ~k3 & ((wb & (ha < TH)) | (wa & (hb < TH)))
        k1 = open_ & ~k2 & ~k3 & ~k4
        zero = torch.zeros_like(ha)
        f = torch.where(k2 & wa, 0.5440 * ha * torch.sqrt(G * ha), zero)
        f = torch.where(k3 & wb, -0.544 * hb * torch.sqrt(G * hb), f)
        hh3 = torch.maximum(eb, ea) - torch.maximum(zb, za)
        sgn = torch.where((hb - TH) - (ha - TH) >= 0, 1.0, -1.0).to(ha.dtype)
        f = torch.where(k4, -sgn * 0.350 * hh3 * torch.sqrt((2.0 * G * hh3).clamp_min(0.0)), f)
        return k1, f, eb - ea

    def momentum(self, q0, u0, vt, hm, deta, conv, nf, dt2, dt2n):
        ram = torch.where(hm > TH, G * nf * nf * torch.sqrt(u0 * u0 + vt * vt) / hm.clamp_min(TH).pow(1.3333330),
                          torch.zeros_like(hm))
        a = 0.5 * dt2 * ram
        return ((1.0 - a) * q0 - conv - G * hm * dt2n * deta) / (1.0 + a)

    def flux(self, dt2):
        c, at = self.c, self.at
        dtn = dt2 / c["dx"]
        H, Z, A, N = self.pad(self.h), self.pad(self.z), self.pad(self.act), self.pad(self.n)
        qx, qy, u, v = self.qx, self.qy, self.u, self.v

        def edge(w1, w0, q0, q1):
            a = 0.5 * (w1 + w0)
            return 0.5 * (a * (q1 + q0) + a.abs() * (q0 - q1))

        hb, zb, nb, ab = at(H), at(Z), at(N), at(A)
        # x faces: north of the cell
        ha, za = at(H, -1), at(Z, -1)
        k1, F, de = self.special(ha, hb, za, zb, ab & at(A, -1))
        along = edge(at(u, 1), at(u), at(qx), at(qx, 1)) - edge(at(u), at(u, -1), at(qx, -1), at(qx))
        cross = (edge(at(v, 0, 1), at(v, -1, 1), at(qx), at(qx, 0, 1))
                 - edge(at(v), at(v, -1), at(qx, 0, -1), at(qx)))
        cross[:, 0] = 0.0
        vt = 0.25 * (at(v) + at(v, 0, 1) + at(v, -1) + at(v, -1, 1))
        Fm = self.momentum(at(qx), at(u), vt, 0.5 * (ha + hb), de, dtn * (along + cross), 0.5 * (nb + at(N, -1)), dt2, dtn)
        fx = torch.where(k1, Fm, F)
        if c["outflow"]:
            hw = self.h[-1]
            fx[self.R, :self.C] = torch.where(self.act[-1] & (hw > TH), 0.5440 * hw * torch.sqrt(G * hw), torch.zeros_like(hw))
        # y faces: west of the cell
        ha, za = at(H, 0, -1), at(Z, 0, -1)
        k1, F, de = self.special(ha, hb, za, zb, ab & at(A, 0, -1))
        along = edge(at(v, 0, 1), at(v), at(qy), at(qy, 0, 1)) - edge(at(v), at(v, 0, -1), at(qy, 0, -1), at(qy))
        cross = (edge(at(u, 1), at(u, 1, -1), at(qy), at(qy, 1))
                 - edge(at(u), at(u, 0, -1), at(qy, -1), at(qy)))
        cross[0] = 0.0
        ut = 0.25 * (at(u) + at(u, 1) + at(u, 0, -1) + at(u, 1, -1))
        Fm = self.momentum(at(qy), at(v), ut, 0.5 * (ha + hb), de, dtn * (along + cross), 0.5 * (nb + at(N, 0, -1)), dt2, dtn)
        return fx, torch.where(k1, Fm, F)

    def depth(self, fx, fy, dt2, t):
        c, d = self.c, self.d
        per = d["dtrain"] * 1000.0
        rain = _series(d["rain"], d["dtrain"], t, c["series"]) / per
        evap = _series(d["evap"], d["dtrain"], t, c["series"]) / per if d["evap"] is not None else 0.0
        fi, ff, fl = d["frac"]
        lake = self.h > EV_WL_MIN
        like = lambda a: torch.full_like(self.h, a)  # noqa: E731
        pct = torch.where(lake, like(1.0 - fl), like(1.0 - (fi + ff)))
        R, C = self.R, self.C
        s = (fx[1:R + 1, :C] - fx[:R, :C]) / c["dx"] + (fy[:R, 1:C + 1] - fy[:R, :C]) / c["dx"]
        if d["src"] is not None:
            for k, cell in enumerate(d["src"]):
                q = _series(d["srcq"][:, k], 3600.0, t, c["series"]) / self.area
                s[int(cell) // C, int(cell) % C] -= q
        s = s - (rain * self.w if self.w is not None else rain) * pct
        if evap:
            s = s + torch.where(lake, like(evap), like(0.0))
        h = (self.h - dt2 * s).clamp_min(0.0)
        return torch.where(self.act, h, torch.zeros_like(h))

    def iterate(self, dt2, tm):
        R, C = self.R, self.C
        fx, fy = self.flux(dt2)
        dry = self.act & (self.depth(fx, fy, dt2, self.t) < TH)
        D = self.pad(dry)
        c_, n_, w_ = self.at(D), self.at(D, -1), self.at(D, 0, -1)
        fx = torch.where(((fx > 0) & n_) | ((fx < 0) & c_), torch.zeros_like(fx), fx)
        fy = torch.where(((fy > 0) & w_) | ((fy < 0) & c_), torch.zeros_like(fy), fy)
        hn = self.depth(fx, fy, dt2, tm)
        self.S = self.speed()  # of the state this iteration started from
        self.h = hn
        fx[:, C] = 0.0
        fy[R] = 0.0
        hx = torch.cat([hn[:1], 0.5 * (hn[1:] + hn[:-1]), hn[-1:]])
        hy = torch.cat([hn[:, :1], 0.5 * (hn[:, 1:] + hn[:, :-1]), hn[:, -1:]], dim=1)
        u, v = torch.zeros_like(fx), torch.zeros_like(fy)
        u[:, :C] = torch.where(hx >= TH, fx[:, :C] / hx.clamp_min(TH), torch.zeros_like(hx))
        v[:R] = torch.where(hy >= TH, fy[:R] / hy.clamp_min(TH), torch.zeros_like(hy))
        self.qx, self.qy, self.u, self.v = self.put(fx), self.put(fy), self.put(u), self.put(v)

    def run(self):
        c = self.c
        t_end = c["seconds"] if c["advance"] else math.inf
        n = 0
        while n < (10 ** 9 if c["advance"] else c["iters"]):
            if c["dt_mode"] == "fixed":
                if not self.t + c["dt"] <= t_end:
                    break
                tm = self.t + c["dt"]
                dt2, nxt = 2.0 * c["dt"], tm + c["dt"]
            else:
                if not self.t < t_end:
                    break
                dt2 = min(2.0, 0.7 / self.S) if self.S > 0 else 2.0
                dt2 = min(dt2, t_end - self.t)
                tm, nxt = self.t + 0.5 * dt2, self.t + dt2
            self.iterate(dt2, tm)
            self.t = nxt
            n += 1


def _velocity64(s):
    """Cell velocities."""
    R, C = s.R, s.C
    u, v = s.u[2:3 + R, 2:2 + C], s.v[2:2 + R, 2:3 + C]
    wet = s.h >= TH
    zero = torch.zeros_like(s.h)
    return torch.where(wet, 0.5 * (u[1:] + u[:-1]), zero), torch.where(wet, 0.5 * (v[:, 1:] + v[:, :-1]), zero)


def _smooth64(m, z):
    """The lake edge's cells in the sweep's order (south row first, west to east), each the mean of its two
    neighbours across the edge, updated in place."""
    i = m[1:-1, 1:-1]
    edge = (i != 1) & ((i != m[:-2, 1:-1]) | (i != m[2:, 1:-1]) | (i != m[1:-1, :-2]) | (i != m[1:-1, 2:]))
    for r, c in sorted((np.argwhere(edge) + 1).tolist(), key=lambda p: (-p[0], p[1])):
        for a, b in (((r - 1, c), (r + 1, c)), ((r + 1, c), (r - 1, c)), ((r, c - 1), (r, c + 1)), ((r, c + 1), (r, c - 1))):
            if m[r, c] != m[a] and z[b] != NODATA:
                z[r, c] = (z[a] + z[b]) / 2.0
    return z


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "batch":
        return None
    if c["kind"] == "lake":
        st = prepare(c, seed)
        return _smooth64(st["mask"].cpu().numpy(), st["dem"].cpu().numpy())
    if c["kind"] == "measure":
        z, h, qx, qy = _measure_inputs(c, seed)
        act = z != NODATA
        speed = 0.0
        for dim, q in ((0, qx[1:-1]), (1, qy[:, 1:-1])):
            n = h.shape[dim]
            hm = 0.5 * (h.narrow(dim, 1, n - 1) + h.narrow(dim, 0, n - 1))
            ok = act.narrow(dim, 1, n - 1) & act.narrow(dim, 0, n - 1) & (hm >= TH)
            s = (q / hm.clamp_min(TH)).abs() + torch.sqrt(G * hm)
            speed += float(torch.where(ok, s / c["dx"], torch.zeros_like(s)).max())
        return float(torch.where(act, h, torch.zeros_like(h)).sum()) * c["dx"] ** 2, speed
    d = _inputs(c, seed)
    s = _Step64(c, d)
    s.run()
    R, C = s.R, s.C
    out = {"t": s.t, "depth": s.h}
    if c["read"] != "depth":
        out["qx"], out["qy"] = s.qx[2:3 + R, 2:2 + C], s.qy[2:2 + R, 2:3 + C]
    if c["couple"]:
        out["uu"], out["vv"] = _velocity64(s)
        out["boundary"] = None
    return out
