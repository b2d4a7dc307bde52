"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case is one pass through the public entry points on a seeded scenario
of the package's own generators (a planar shelf with a granular cap, or a
spherical fjord with dry land): a forecast, a batch of scenarios, a gradient.
"swell" cases start from a sea in motion (long waves and their discharges on
every wet cell), "rest" cases from still water above a slide, as a run begins.

``exact`` restates the scheme in plain torch in 64 bits (autograd for the
gradients), on whole fields instead of per edge and per cell.
"""
import ctypes
import math

import numpy as np
import torch

from landslidehysea_gb300 import scenarios
from landslidehysea_gb300._abi import VARS
from landslidehysea_gb300.solver import Adjoint, AdjointBatch, Batch, Solver, load

PARAMS = ("angle1", "mf0", "mfs", "r")
FJORD_CELL = 0.0002 * 2048  # degrees across the fjord's domain: smaller grids keep the domain, dry land included


# ---------------------------------------------------------------- the cases
def listed():
    def shelf(name, nx, ny, **kw):
        return {"name": name, "scene": "shelf", "nx": nx, "ny": ny, "start": "swell", **kw}

    def fjord(name, n, **kw):
        return {"name": name, "scene": "fjord", "nx": n, "ny": n, "start": "swell", **kw}

    return [
        # the smallest grids: what a first trial, a unit test or a 1-D-like check of a setup runs; launches and latency
        shelf("solve_o1_24x17", 24, 17, do="solve", order=1, steps=32),
        fjord("solve_o2_64", 64, do="solve", order=2, steps=32),
        # the reference's own example size, from rest, as its run begins (first order, Cartesian)
        shelf("solve_o1_200", 200, 200, do="solve", order=1, steps=100, start="rest"),
        # a ragged grid with the options that site studies switch on: Pouliquen friction, speed caps, interlayer
        # friction, open boundaries, the tracked maximum of the free surface
        shelf("solve_o1_options_331x217", 331, 217, do="solve", order=1, steps=32, options=True),
        # an ordinary regional grid, odd size, second order, spherical
        fjord("solve_o2_523", 523, do="solve", order=2, steps=24),
        # the headline: the 2048 x 2048 second-order spherical fjord from rest
        fjord("solve_o2_2048", 2048, do="solve", order=2, steps=24, start="rest"),
        # the largest all-wet grid: open sea, first order
        shelf("solve_o1_2048", 2048, 2048, do="solve", order=1, steps=8),
        # a warning-centre run: host arrays in, gauge readings at intervals of simulated time, fields and maxima out
        fjord("forecast_o2_512", 512, do="forecast", order=2, readings=6, every=8),
        # a coupled host that owns all device memory and exchanges data after every step
        shelf("noalloc_o1_160x96", 160, 96, do="noalloc", order=1, steps=8),
        # an ensemble over friction angle, density ratio and slide volume, on uneven grids
        {"name": "ensemble_o2_10", "do": "ensemble", "scene": "shelf", "count": 10, "lo": 128, "hi": 512, "order": 2,
         "steps": 40, "start": "swell"},
        # a gradient for source and friction inversion against gauges
        fjord("gradient_o2_1024", 1024, do="gradient", order=2, steps=24),
        # a calibration: several scenarios' gradients under one joint checkpoint budget that has steps recomputed
        {"name": "calibration_o2_6", "do": "calibration", "scene": "fjord", "count": 6, "lo": 96, "hi": 384, "order": 2,
         "steps": 6, "slots": 3, "start": "swell"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["solve", "solve", "solve", "forecast", "noalloc", "ensemble", "gradient", "calibration"])
    order = rng.choice([1, 2])
    scene = rng.choice(["shelf", "fjord"])
    start = rng.choice(["swell", "swell", "rest"])
    case = {"do": do, "scene": scene, "order": order, "start": start}
    if do == "solve":
        nx = size(16, 1800)
        ny = nx if scene == "fjord" else max(8, min(1800, int(nx * rng.uniform(0.4, 2.0))))
        return {**case, "nx": nx, "ny": ny, "steps": rng.randint(6, 40) if nx * ny < 300_000 else rng.randint(3, 8),
                "options": scene == "shelf" and rng.random() < 0.4}
    if do == "forecast":
        n = size(48, 700)
        return {**case, "nx": n, "ny": n, "readings": rng.randint(2, 8), "every": rng.randint(2, 12)}
    if do == "noalloc":
        nx, ny = size(16, 250), size(16, 250)
        return {**case, "scene": "shelf", "order": 1, "nx": nx, "ny": ny, "steps": rng.randint(2, 16)}
    if do == "ensemble":
        lo = size(24, 200)
        return {**case, "count": rng.randint(2, 10), "lo": lo, "hi": min(512, int(lo * rng.uniform(1.0, 3.0))),
                "steps": rng.randint(4, 24)}
    # gradients start from a sea in motion: at rest many cells tie for the time step's arg-max
    if do == "gradient":
        n = size(24, 500)
        return {**case, "nx": n, "ny": n, "steps": rng.randint(3, 8), "start": "swell"}
    lo = size(24, 120)
    return {**case, "count": rng.randint(2, 6), "lo": lo, "hi": int(lo * rng.uniform(1.0, 2.5)),
            "steps": rng.randint(3, 6), "slots": rng.randint(2, 4), "start": "swell"}


# ---------------------------------------------------------------- inputs
def _sizes(case):
    """(nx, ny) of each scenario of a case."""
    if "count" not in case:
        return [(case["nx"], case["ny"])]
    n, lo, hi = case["count"], case["lo"], case["hi"]
    return [(v, v) for v in (int(round(lo * (hi / lo) ** (k / max(1, n - 1)))) for k in range(n))]


def _swell(state, p, rng):
    """Long waves of up to half a metre on the wet cells, with their discharges (a progressive wave's u = eta sqrt(g/h))."""
    ny, nx = state["h1"].shape
    y = np.arange(ny)[:, None] / max(ny, 2)
    x = np.arange(nx)[None, :] / max(nx, 2)
    eta = np.zeros((ny, nx))
    for _ in range(3):
        kx, ky = rng.uniform(-6.0, 6.0, 2)
        eta += np.sin(2.0 * math.pi * (kx * x + ky * y) + rng.uniform(0.0, 2.0 * math.pi))
    h1 = state["h1"]
    eta *= (0.5 / 3.0) * np.minimum(1.0, h1 / 5.0)
    th = rng.uniform(0.0, 2.0 * math.pi)
    h = h1 + np.where(h1 > 0.0, eta, 0.0)
    q = eta * np.sqrt(p.gravity * h)
    return {**state, "h1": h, "q1x": q * math.cos(th), "q1y": q * math.sin(th)}


def _scene(case, nx, ny, seed):
    """(parameters, state, flat gauge cells) of one scenario."""
    rng = np.random.default_rng(seed)
    o2 = case["order"] == 2
    if case["scene"] == "fjord":
        sc = scenarios.fjord(n=nx, seed=seed, dcell_deg=FJORD_CELL / nx, order=case["order"], cfl=0.5 if o2 else 0.9)
        sc.params.eig_sort = 1 if nx % 2 else 0
        gauges = scenarios.gauge_cells(sc)
    else:
        sc = scenarios.shelf(nx=nx, ny=ny, seed=seed, dx=max(25.0, 5000.0 / nx), order=case["order"], cfl=0.5 if o2 else 0.9,
                             angle_deg=rng.uniform(8.0, 20.0), r=rng.uniform(0.45, 0.6),
                             cap_volume=math.exp(rng.uniform(math.log(1e6), math.log(1e8))))
        gauges = np.sort(rng.choice(nx * ny, min(16, nx * ny), replace=False)).astype(np.int32)
    p = sc.params
    if case.get("options"):
        p.friction_law, p.track_eta_max, p.mfc, p.vmax1, p.vmax2 = 1, 1, 0.01, 20.0, 15.0
        p.angle2, p.angle3, p.angle4 = p.angle1 * 1.5, p.angle1 * 1.1, p.angle1 * 1.6
        p.borde_sup = p.borde_inf = p.borde_izq = p.borde_der = 1.0
    if case["do"] == "forecast":
        p.track_eta_max = 1
    state = _swell(sc.state, p, rng) if case["start"] == "swell" else sc.state
    return p, {v: np.ascontiguousarray(state[v], dtype=np.float64) for v in VARS}, gauges


def _scenes(case, seed):
    return [_scene(case, nx, ny, 1000 * seed + k) for k, (nx, ny) in enumerate(_sizes(case))]


def _interval(case):
    """Simulated seconds between a forecast's readings: about "every" steps of a grid of this size."""
    dt = 0.068 * 2048 / case["nx"] if case["scene"] == "fjord" else 0.5 * max(25.0, 5000.0 / case["nx"]) / 50.0
    return case["every"] * dt


def _targets(case, scenes, seed):
    """Observed series: the level at rest or swell that the gauges start from, and 0.3 m of signal."""
    rng = np.random.default_rng(seed)
    first = [(st["h1"] + st["h2"] - st["H"]).reshape(-1)[g] for _, st, g in scenes]
    return [e + 0.3 * rng.standard_normal((case["steps"], e.size)) for e in first]


def prepare(case, seed):
    scenes = _scenes(case, seed)
    p, state, gauges = scenes[0]
    s = {"case": case, "scenes": scenes}
    do = case["do"]
    if do in ("solve", "noalloc"):
        s["in"] = torch.from_numpy(np.stack([state[v] for v in VARS])).cuda()
        s["out"] = torch.empty_like(s["in"])
        s["in_ptrs"], s["out_ptrs"] = ([a.data_ptr() for a in s[k]] for k in ("in", "out"))
    if do in ("solve", "forecast"):
        s["solver"] = Solver(p)
    if do == "forecast":
        s["host"] = np.empty((len(VARS), p.ny, p.nx))
    if do == "ensemble":
        s["batch"] = Batch([sc[0] for sc in scenes])
    if do in ("gradient", "calibration"):
        s["targets"] = _targets(case, scenes, seed)
    if do == "gradient":
        s["adjoint"] = Adjoint(p, gauges)
        s["adjoint"].set_thin_layer(0.1)
    if do == "calibration":
        s["adjoint"] = AdjointBatch([sc[0] for sc in scenes], [sc[2] for sc in scenes])
        s["adjoint"].set_thin_layer(0.1)
        s["adjoint"].set_budget(case["slots"] * sum(48.0 * (-(-nx * ny // 32) * 32) for nx, ny in _sizes(case)))
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    return {"solve": _solve, "forecast": _forecast, "noalloc": _noalloc, "ensemble": _ensemble, "gradient": _gradient,
            "calibration": _calibration}[s["case"]["do"]](s)


def _solve(s):
    """The state from device arrays, a run of steps, the state back into device arrays."""
    c = s["solver"]
    c.set_state_device(s["in_ptrs"])
    c.step(s["case"]["steps"])
    c.get_state_device(s["out_ptrs"])
    c.synchronize()
    out = {"state": s["out"]}
    if s["case"].get("options"):
        out["eta_max"], out["eta_time"] = c.eta_max()
    return out


def _forecast(s):
    c, case, (p, state, gauges) = s["solver"], s["case"], s["scenes"][0]
    c.set_state(state)
    series = []
    for k in range(case["readings"]):
        c.run_until((k + 1) * _interval(case))
        series.append(c.gauge_eta(gauges))
    em, et = c.eta_max()
    c.get_state(out=dict(zip(VARS, s["host"])))
    return {"state": s["host"], "eta_max": em, "eta_time": et, "series": series}


def _noalloc(s):
    lib, p = load(), s["scenes"][0][0]
    s["out"].copy_(s["in"])
    ptrs = (ctypes.c_void_p * len(VARS))(*s["out_ptrs"])
    t, dt = ctypes.c_double(0.0), ctypes.c_double(0.0)
    for _ in range(s["case"]["steps"]):
        if lib.lsh_step_noalloc(ctypes.byref(p), ptrs, 1, ctypes.byref(t), ctypes.byref(dt), None):
            raise RuntimeError("lsh_step_noalloc failed")
    return {"state": s["out"], "time": t.value, "dt": dt.value}


def _ensemble(s):
    b = s["batch"]
    for k, (_, state, _) in enumerate(s["scenes"]):
        b.set_state(k, state)
    b.step(s["case"]["steps"])
    b.synchronize()
    return [{v: a for v, a in b.get_state(k).items() if v != "H"} for k in range(len(s["scenes"]))]


def _gradient(s):
    a = s["adjoint"]
    misfit, series = a.forward(s["scenes"][0][1], s["case"]["steps"], s["targets"][0])
    g, gp = a.gradient()
    return {"misfit": misfit, "series": series, "state": g, "params": np.array([gp[k] for k in PARAMS])}


def _calibration(s):
    a = s["adjoint"]
    misfits, series = a.forward([sc[1] for sc in s["scenes"]], s["case"]["steps"], s["targets"])
    g, gp = a.gradient()
    return {"misfits": misfits, "series": series, "state": g, "params": np.array([[d[k] for k in PARAMS] for d in gp])}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """The fields in and out once, and the scheme's operations on the wet cells (380 a cell and step at first order, 804
    at second; a gradient replays each step and reverses it at about 2.5 times its cost)."""
    cells = sum(nx * ny for nx, ny in _sizes(case))
    do = case["do"]
    steps = case["readings"] * case["every"] if do == "forecast" else case["steps"]
    wet = 0.14 if case["scene"] == "fjord" else 1.0
    flops = cells * wet * steps * (380.0 if case["order"] == 1 else 804.0)
    arrays = 7 + 6  # the state in, the state (or its gradient) out
    if do == "forecast" or case.get("options"):
        arrays += 2
    if do in ("gradient", "calibration"):
        flops *= 4.5
    return {"bytes": 8.0 * arrays * cells, "flops": flops}


# ---------------------------------------------------------------- the same numbers in plain torch, 64 bits
EPS = 1.1920928955078125e-07  # the scheme's EPSILON
ROOT2 = 1.41421356237309504880


def _w(c, a, b):
    if not torch.is_tensor(a):
        a = torch.full_like(b, a) if torch.is_tensor(b) else torch.tensor(a, dtype=torch.float64, device=c.device)
    if not torch.is_tensor(b):
        b = torch.full_like(a, b)
    return torch.where(c, a, b)


def _max0(x):
    return _w(x > 0, x, 0.0)


def _min(a, b):
    return _w(b < a, b, a)


def _max(a, b):
    return _w(a < b, b, a)


def _abs(x):
    return _w(x < 0, -x, x)


def _sqrt(x):
    c = x > 0
    return _w(c, torch.sqrt(_w(c, x, 1.0)), 0.0)


def _inv(x, use):
    return 1.0 / _w(use, x, 1.0)


class _Scheme:
    """The two-layer scheme of one parameter set: path-conservative IFCP edges in four colour passes, cell update with
    filter, friction and Coulomb stop; at second order minmod faces and Heun's method.  Fields are [ny, nx] tensors."""

    def __init__(self, p, dev, par=None):
        f = dict(dtype=torch.float64, device=dev)
        self.p, self.f = p, f
        par = torch.tensor([getattr(p, k) for k in PARAMS], **f) if par is None else par
        angle1, mf0, mfs, self.r = par.unbind()
        self.eps, self.g = p.eps_h, p.gravity
        self.gp = p.gravity * (1.0 - self.r)
        self.tan = [torch.tan(angle1)] + [math.tan(a) for a in (p.angle2, p.angle3, p.angle4)]
        self.mu = _abs(self.tan[0]) * (p.L / p.H)
        self.g_mf02, self.g_mfs2 = p.gravity * mf0 * mf0, p.gravity * mfs * mfs
        j = np.arange(p.ny)
        if p.coords:
            d = math.pi / 180.0
            R, dl, dp = p.radius, p.dlon * d, p.dlat * d
            lat = (p.lat0 + np.arange(p.ny + 1) * p.dlat) * d
            mid = (p.lat0 + (j + 0.5) * p.dlat) * d
            area = R * R * dl * (np.sin((p.lat0 + (j + 1) * p.dlat) * d) - np.sin((p.lat0 + j * p.dlat) * d))
            geo = (area, np.full(p.ny, R * dp), R * np.cos(lat) * dl, np.tan(mid) / R, area / (R * np.cos(mid) * dl),
                   area / (R * dp))
        else:
            one = np.ones(p.ny)
            geo = (p.dx * p.dy * one, p.dy * one, p.dx * np.ones(p.ny + 1), 0.0 * one, p.dy * one, p.dx * one)
        self.area, self.len_v, self.len_h, self.tanR, self.wx, self.wy = (torch.tensor(a, **f)[:, None] for a in geo)

    def vfac(self, h):
        wet = h > self.eps
        low = _w(wet, 0.0, h)
        return _w(wet, _inv(h, wet), ROOT2 * low / torch.sqrt(low ** 4 + self.eps ** 4))

    def fsc(self, h1):
        a = 10.0 * h1 / self.eps
        return 1.0 - self.r * (1.0 - torch.exp(-(a * a)))

    def friction(self, h1, u1, h2, u2):
        if self.p.friction_law == 0:
            return self.mu
        t, beta, l2, chi = self.tan, 0.136, 8.0e-4, 1.0e-3
        rr = self.fsc(h1)
        gp = self.g * rr
        fr1, fr2 = u1 * u1 * self.vfac(h1) / gp, u2 * u2 * self.vfac(h2) / gp
        fr = _sqrt(fr1 + fr2 + (1.0 - rr) * fr1 * fr2)
        den = 1.0 + h2 / l2
        stop, start = t[0] + (t[1] - t[0]) / den, t[2] + (t[3] - t[2]) / den
        fast, slow = fr > beta, fr < EPS
        frs = _w(slow, 1.0, fr)
        mu = _w(fast, t[0] + (t[1] - t[0]) / (1.0 + beta * h2 / (frs * l2)),
                _w(slow, start, torch.pow(frs / beta, chi) * (stop - start) + start))
        return mu * self.p.L / self.p.H

    def eig(self, h1, h2, u1, u2, q):
        h = h1 + h2
        F = self.vfac(h)
        u, cg = q * F, _sqrt(self.g * h)
        uu = (u1 * h2 + u2 * h1) * F
        ci = _sqrt(self.gp * h1 * h2 * F * _abs(1.0 - (u1 - u2) ** 2 * F / self.gp))
        d = [u - cg, uu - ci, uu + ci, u + cg]
        for a, b in ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (1, 2) if self.p.eig_sort else (2, 1), (2, 3)):
            swap = d[a] > d[b]
            d[a], d[b] = _w(swap, d[b], d[a]), _w(swap, d[a], d[b])
        return d

    def roe(self, A, B):
        """Face factors and the Roe averages of one layer's (depth, discharge) pairs."""
        fa, fb = self.vfac(A[0]), self.vfac(B[0])
        sa, sb = _sqrt(A[0]), _sqrt(B[0])
        return fa, fb, (sa * fa * A[1] + sb * fb * B[1]) / (sa + sb + EPS)

    def flux(self, A, B, ln, area, hc, acc, inside, dt):
        """One colour of edges; A, B: faces (h1, qn1, qt1, h2, qn2, qt2, H).  -> (minus, plus, wave)."""
        eps, g, r = self.eps, self.g, self.r
        one = (A[3] == 0) & (B[3] == 0) & (A[4] == 0) & (B[4] == 0)  # no granular layer: no sensitivity to it either
        A, B = list(A), list(B)
        for k in (3, 4, 5):
            A[k], B[k] = _w(one, A[k].detach(), A[k]), _w(one, B[k].detach(), B[k])
        a1, aq1, at1, a2, aq2, at2, H0 = A
        b1, bq1, bt1, b2, bq2, bt2, H1 = B
        h1, h2 = 0.5 * (a1 + b1), 0.5 * (a2 + b2)
        wet = (h1 >= EPS) | (h2 >= EPS)
        bq2 = _w((a2 < eps) & (H1 - b2 > H0), 0.0, bq2)
        aq2 = _w((b2 < eps) & (H0 - a2 > H1), 0.0, aq2)
        bq1 = _w((a1 < eps) & (H1 - b1 - b2 > H0 - a2), 0.0, bq1)
        aq1 = _w((b1 < eps) & (H0 - a1 - a2 > H1 - b2), 0.0, aq1)
        c = (a2 + a1 < eps) & (H1 - b1 - b2 > H0)
        bq1, bq2 = _w(c, 0.0, bq1), _w(c, 0.0, bq2)
        c = (b2 + b1 < eps) & (H0 - a1 - a2 > H1)
        aq1, aq2 = _w(c, 0.0, aq1), _w(c, 0.0, aq2)
        fa1, fb1, u1 = self.roe((a1, aq1), (b1, bq1))
        fa2, fb2, u2 = self.roe((a2, aq2), (b2, bq2))
        Hm = _min(H0, H1)
        de1 = _max0(b1 + b2 - H1 + Hm) - _max0(a1 + a2 - H0 + Hm)
        de2 = _max0(b2 - H1 + Hm) - _max0(a2 - H0 + Hm)
        p1 = g * h1 * de1
        p2 = g * h2 * ((1.0 - r) * de2 + r * de1)
        stop = _abs(h2 * u2) < self.p.peso * self.fsc(h1) * self.friction(h1, u1, h2, u2) * g * h2 * dt
        D = self.eig(h1, h2, u1, u2, h1 * u1 + h2 * u2)
        E0 = self.eig(a1, a2, fa1 * aq1, fa2 * aq2, aq1 + aq2)
        E1 = self.eig(b1, b2, fb1 * bq1, fb2 * bq2, bq1 + bq2)
        l1, l3 = _min(D[0], _min(E0[0], E1[0])), _max(D[3], _max(E0[3], E1[3]))
        lmax = _max(_max(_abs(l3), _abs(l1)), _max(_abs(u1), _abs(u2)))
        l2 = _max(_abs(D[1]), _abs(D[2]))
        l2 = _w((l1 + l3 < 0) & (_abs(l1 + l3) >= EPS), -l2, l2)
        apart = (_abs(l1 - l3) >= EPS) & (_abs(l1 - l2) >= EPS) & (_abs(l2 - l3) >= EPS)
        both = apart & (h1 >= eps) & (h2 >= eps)
        d12, d13, d23 = l1 - l2, l1 - l3, l2 - l3
        inv = _inv(d12 * d13 * d23, both)
        ca, cb, cc = _abs(l1) * d23 * inv, -_abs(l2) * d13 * inv, _abs(l3) * d12 * inv
        inv = _inv(l3 - l1, apart)
        k0 = _w(both, ca * l2 * l3 + cb * l1 * l3 + cc * l1 * l2, _w(apart, (l3 * _abs(l1) - l1 * _abs(l3)) * inv, lmax))
        k1 = _w(both, -(ca * (l2 + l3) + cb * (l1 + l3) + cc * (l1 + l2)), _w(apart, (_abs(l3) - _abs(l1)) * inv, 0.0))
        k2 = _w(both, ca + cb + cc, 0.0)
        fay, fby = _w(a1 < EPS, 0.0, fa1 * aq1 * aq1), _w(b1 < EPS, 0.0, fb1 * bq1 * bq1)
        faw, fbw = _w(a2 < EPS, 0.0, fa2 * aq2 * aq2), _w(b2 < EPS, 0.0, fb2 * bq2 * bq2)
        dx, dy, dz, dw = bq1 - aq1, fby - fay, bq2 - aq2, fbw - faw
        ty = p1 + dy
        tw = _w(stop, g * h2 * r * de1, p2) + dw
        ay = g * h1 * dz + 2.0 * u1 * ty + (g * h1 - u1 * u1) * dx
        aw = r * g * h2 * dx + (g * h2 - u2 * u2) * dz + 2.0 * u2 * tw
        i0 = _w(~stop & (a1 > eps) & (b1 > eps), de1 - de2, de1)
        i2 = _w(stop, 0.0, de2)
        Q = [0.5 * (k0 * i0 + k1 * dx + k2 * ty), 0.5 * (k0 * dx + k1 * ty + k2 * ay),
             0.5 * (k0 * i2 + k1 * dz + k2 * tw), 0.5 * (k0 * dz + k1 * tw + k2 * aw)]
        half = [0.5 * dx, 0.5 * (dy + p1), 0.5 * dz, 0.5 * (dw + p2)]
        M, P = [None] * 6, [None] * 6
        for l, (fa, fb, at, bt, aq, bq, F0, F1) in enumerate(((fa1, fb1, at1, bt1, aq1, bq1, fay, fby),
                                                              (fa2, fb2, at2, bt2, aq2, bq2, faw, fbw))):
            m, pl = half[2 * l] + (aq - Q[2 * l]), half[2 * l] + (Q[2 * l] - bq)
            ut = _w(_abs(m) < EPS, 0.0, _w(m > 0, fa * at, fb * bt))
            mm = [m, half[2 * l + 1] + (F0 - Q[2 * l + 1]), m * ut]
            pp = [pl, half[2 * l + 1] + (Q[2 * l + 1] - F1), -m * ut]
            mm, pp = [ln * v for v in mm], [ln * v for v in pp]
            # positivity limiter on the partial sums
            oa, ob = mm[0] > 0, inside & (pp[0] > 0)
            ha = (hc[0][l] + dt / area[0] * acc[0][l]) * area[0]
            hb = (hc[1][l] + dt / area[1] * acc[1][l]) * area[1]
            da, db = _w(oa, self.p.beta * mm[0] + EPS, 1.0), _w(ob, self.p.beta * pp[0] + EPS, 1.0)
            lim = (oa & (ha < dt * da)) | (ob & (hb < dt * db))
            al = _w(lim, _min(_w(oa, ha / da, 1e30), _w(ob, hb / db, 1e30)) / (dt + EPS), 1.0)
            M[3 * l:3 * l + 3], P[3 * l:3 * l + 3] = [al * v for v in mm], [al * v for v in pp]
        wave = ln * _w(lmax < eps, lmax + eps, lmax)
        return [_w(wet, v, 0.0) for v in M], [_w(wet, v, 0.0) for v in P], _w(wet, wave, 0.0)

    def colour(self, axis, par, n):
        """The edges of one colour along `axis` (0: between rows, 1: between columns): first and second cell, normal
        sign, interior, boundary factor."""
        p = self.p
        e = torch.arange(par, n + 1, 2, device=self.f["device"])
        lo, hi = ((p.borde_sup, p.borde_inf) if axis == 0 else (p.borde_izq, p.borde_der))
        first, last = (e == 0)[:, None], (e == n)[:, None]
        sg = torch.where(first, -1.0, 1.0).to(torch.float64)
        bor = torch.where(first, lo, hi).to(torch.float64)
        return e, (e - 1).clamp(min=0), e.clamp(max=n - 1), sg, ~(first | last), bor

    def faces(self, axis, W, S, i, sg, normal):
        """Faces of cells `i` on their sg side in the frame of normal sign `normal` (fields with edges along dim 0)."""
        w = [v[i] for v in W]
        if S is not None:
            s = [sg * v[i] for v in S]
            w = [w[0] + (s[0] - s[3]), w[1] + s[1], w[2] + s[2], w[3] + (s[3] + s[6]), w[4] + s[4], w[5] + s[5], w[6] + s[6]]
        if axis == 0:
            return [w[0], normal * w[2], -normal * w[1], w[3], normal * w[5], -normal * w[4], w[6]]
        return [w[0], normal * w[1], normal * w[2], w[3], normal * w[4], normal * w[5], w[6]]

    def edges(self, axis, W, S):
        """Per colour along `axis`: (e, i0, i1, inside, sg, A, B), ghosts at the boundary."""
        t = (lambda v: v) if axis == 0 else (lambda v: v.t())
        W = [t(v) for v in W]
        S = None if S is None else [t(v) for v in S]
        n = W[0].shape[0]
        for par in (0, 1):
            e, i0, i1, sg, inside, bor = self.colour(axis, par, n)
            A = self.faces(axis, W, S, i0, sg, sg)
            B = self.faces(axis, W, S, i1, -1.0, sg)
            ghost = [A[0], A[1] * bor, A[2], A[3], A[4] * bor, A[5], A[6]]
            yield W, e, i0, i1, inside, sg, A, [_w(inside, b, gh) for b, gh in zip(B, ghost)]

    def slopes(self, W):
        h1, h2, H = W[0], W[3], W[6]
        out = []
        v = [h1 + h2 - H, W[1], W[2], h2 - H, W[4], W[5], H]
        for axis in (1, 0):
            s = []
            for q in v:
                q = q if axis == 0 else q.t()
                z = torch.zeros_like(q)
                if q.shape[0] > 2:
                    d = q[1:] - q[:-1]
                    a, b = d[:-1], d[1:]
                    up = _w((a > 0) & (b > 0), _w(a < b, a, b), _w((a < 0) & (b < 0), _w(a > b, a, b), 0.0))
                    z = torch.cat([z[:1], 0.5 * up, z[:1]])
                s.append(z if axis == 0 else z.t())
            out.append(s)
        bad = torch.zeros_like(h1, dtype=torch.bool)
        for s in out:
            for h, d in ((h1, s[0] - s[3]), (h2, s[3] + s[6])):
                bad = bad | (h + d < 0.5 * h) | (h - d < 0.5 * h)
        return [[_w(bad, 0.0, q) for q in s] for s in out]

    def stage(self, W, dt):
        """One Euler stage: (new fields, time step that its wave speeds allow)."""
        p = self.p
        S = self.slopes(W) if p.order == 2 else (None, None)
        acc = [torch.zeros_like(W[0]) for _ in range(7)]
        for axis in (0, 1):
            for Wt, e, i0, i1, inside, sg, A, B in self.edges(axis, W, S[1 - axis]):
                t = (lambda v: v) if axis == 0 else (lambda v: v.t())
                ln = self.len_h[e] if axis == 0 else self.len_v.t()
                area = (self.area[i0], self.area[i1]) if axis == 0 else (self.area.t(), self.area.t())
                ac = [t(v) for v in acc]
                M, P, wave = self.flux(A, B, ln, area, ((Wt[0][i0], Wt[3][i0]), (Wt[0][i1], Wt[3][i1])),
                                       ((ac[0][i0], ac[3][i0]), (ac[0][i1], ac[3][i1])), inside, dt)
                k = inside[:, 0]
                for d, i, sel in ((M, i0, None), (P, i1, k)):
                    for l in (0, 3):
                        xy = (d[l], -sg * d[l + 2], sg * d[l + 1]) if axis == 0 else (d[l], sg * d[l + 1], sg * d[l + 2])
                        for q in range(3):
                            v = xy[q] if sel is None else xy[q][sel]
                            ac[l + q] = ac[l + q].index_add(0, i if sel is None else i[sel], -v)
                    ac[6] = ac[6].index_add(0, i if sel is None else i[sel], wave if sel is None else wave[sel])
                acc = [t(v) for v in ac]
        if p.order == 2:
            for q, s, wgt in ((1, S[0], self.wx), (2, S[1], self.wy)):
                acc[q] = acc[q] - p.peso * (self.g * W[0] * 2.0 * s[0] * wgt)
                acc[q + 3] = acc[q + 3] - p.peso * (self.g * W[3] * 2.0 * ((1.0 - self.r) * s[3] + self.r * s[0]) * wgt)
        return self.cells(W, acc, dt), self.dt_of(acc[6])

    def dt_of(self, wave):
        rate = _w(wave < EPS, 0.0, wave / self.area).reshape(-1)
        top = (rate == rate.max()).nonzero()[0, 0]
        return 2.0 * self.p.cfl / rate[top] if float(rate.detach()[top]) > 0 else torch.tensor(1e30, **self.f)

    def cells(self, W, acc, dt):
        p, eps = self.p, self.eps
        w = [W[k] + dt / self.area * acc[k] for k in range(6)]
        for k in (0, 3):
            s = dt * (self.vfac(W[k]) * W[k + 1] * self.tanR)
            w[k + 1], w[k + 2] = w[k + 1] + s * W[k + 2], w[k + 2] - s * W[k + 1]
        w[0], w[3] = _w(w[0] < 0, 0.0, w[0]), _w(w[3] < 0, 0.0, w[3])
        for k, vmax in ((0, p.vmax1), (3, p.vmax2)):  # filter of thin layers, speed caps
            damp = torch.exp(-dt / ((w[k] / eps) ** 4 + EPS))
            w[k + 1], w[k + 2] = w[k + 1] * damp, w[k + 2] * damp
            if vmax > 0:
                f = self.vfac(w[k])
                u = _sqrt((f * w[k + 1]) ** 2 + (f * w[k + 2]) ** 2)
                fast = u > vmax
                s = vmax * _inv(u, fast)
                for q in (k + 1, k + 2):
                    w[q] = _w(fast, f * w[q] * s * w[k], w[q])
        # bottom and interlayer friction, implicit
        h1, h2 = w[0], w[3]
        f1, f2, o1, o2 = self.vfac(h1), self.vfac(h2), self.vfac(W[0]), self.vfac(W[3])
        speed1 = _sqrt((o1 * W[1]) ** 2 + (o1 * W[2]) ** 2)
        speed2 = _sqrt((o2 * W[4]) ** 2 + (o2 * W[5]) ** 2)
        du = _sqrt((o1 * W[1] - o2 * W[4]) ** 2 + (o1 * W[2] - o2 * W[5]) ** 2)
        p43 = [_w(h > 0, torch.pow(_w(h > 0, h, 1.0), 4.0 / 3.0), 0.0) for h in (h1, h2)]
        both = (h1 > 0) & (h2 > 0)
        hmod = self.r * h1 + h2
        m = _w(hmod > eps * (1.0 + self.r), hmod, eps * (1.0 + self.r))
        k12 = dt * ROOT2 * hmod / torch.sqrt(hmod ** 4 + m ** 4) * p.mfc * du
        c1, c2, c3 = k12 * h2, k12 * self.r * h1, dt * self.g_mfs2 * speed2 / (p43[1] + EPS)
        e1, e2 = 1.0 + c1, 1.0 + c2 + c3
        det = 1.0 / (e1 * e2 - c1 * c2)
        new = list(w)
        for q in (1, 2):
            ua, ub = f1 * w[q], f2 * w[q + 3]
            new[q] = _w(both, h1 * (ua * e2 + c1 * ub) * det, w[q])
            new[q + 3] = _w(both, h2 * (ub * e1 + c2 * ua) * det, w[q + 3])
        for k, alone, sp, gm in ((0, (h1 > 0) & (h2 < eps), speed1, self.g_mf02), (3, (h2 > 0) & (h1 < eps), speed2, self.g_mfs2)):
            y = p43[k // 3] + EPS
            s = y / (y + dt * gm * sp)
            keep = _w(w[k] > eps, 1.0, w[k] * self.vfac(w[k]))
            for q in (k + 1, k + 2):
                new[q] = _w(alone, new[q] * keep * s, new[q])
        # Coulomb stop
        w = new
        n1 = _sqrt(w[1] ** 2 + w[2] ** 2) * self.vfac(w[0])
        n2 = _sqrt(w[4] ** 2 + w[5] ** 2)
        sc = self.fsc(w[0]) * self.friction(w[0], n1, w[3], n2 * self.vfac(w[3])) * self.g * w[3] * dt
        moves = (w[3] > 0) & (n2 + sc >= EPS) & (n2 >= sc)
        aux = _w(moves, n2 * _inv(n2 + sc, moves), 0.0)
        w[4], w[5] = w[4] * aux, w[5] * aux
        return w

    def first_dt(self, W):
        wave = torch.zeros_like(W[0])
        for axis in (0, 1):
            t = (lambda v: v) if axis == 0 else (lambda v: v.t())
            for _, e, i0, i1, inside, sg, A, B in self.edges(axis, W, None):
                h1, h2 = 0.5 * (A[0] + B[0]), 0.5 * (A[3] + B[3])
                u1, u2 = self.roe(A[0:2], B[0:2])[2], self.roe(A[3:5], B[3:5])[2]
                D = self.eig(h1, h2, u1, u2, h1 * u1 + h2 * u2)
                lmax = _max(_max(D[0], D[3]), _max(_abs(u1), _abs(u2)))
                v = (self.len_h[e] if axis == 0 else self.len_v.t()) * _w(lmax < self.eps, lmax + self.eps, lmax)
                k = inside[:, 0]
                wave = t(t(wave).index_add(0, i0, v).index_add(0, i1[k], v[k]))
        return self.dt_of(wave)

    def step(self, W, dt):
        """(fields after one time step, the next time step)."""
        w, nxt = self.stage(W, dt)
        if self.p.order == 2:
            w2, _ = self.stage(w + [W[6]], dt)
            w = [0.5 * (a + b) for a, b in zip(W, w2)]
        return w + [W[6]], nxt


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fields(state):
    return [torch.from_numpy(state[v]).to(_device()) for v in VARS]


def _march(p, state, steps=None, readings=(), gauges=()):
    """Runs `steps` steps, or to each reading's time: (fields, t, dt, eta1 max and its time, gauge rows)."""
    with torch.no_grad():
        sch, W = _Scheme(p, _device()), _fields(state)
        dt, t = sch.first_dt(W), 0.0
        top, when, rows = W[0] + W[3] - W[6], torch.zeros_like(W[0]), []

        def one():
            nonlocal W, dt, t, top, when
            v = W[0] - W[6]
            when, top = torch.where(v > top, t, when), torch.maximum(top, v)
            (W, nxt), t = sch.step(W, dt), t + float(dt)
            dt = nxt

        for _ in range(steps or 0):
            one()
        for end in readings:
            while t < end:
                one()
            rows.append((W[0] - W[6]).reshape(-1)[torch.as_tensor(gauges, dtype=torch.long, device=W[0].device)])
        return W, t, dt, top, when, rows


def _reverse(p, state, gauges, target, steps, thin):
    """(misfit, gauge series, gradient fields, gradient of the parameters) by autograd, one step at a time."""
    dev = _device()
    par = torch.tensor([getattr(p, k) for k in PARAMS], dtype=torch.float64, device=dev, requires_grad=True)
    at = torch.as_tensor(gauges, dtype=torch.long, device=dev)
    tgt = torch.from_numpy(target).to(dev)
    with torch.no_grad():
        sch = _Scheme(p, dev)
        W = _fields(state)
        H = W[6]
        dts, states = [sch.first_dt(W)], [W]
        for _ in range(steps):
            W, nxt = sch.step(W, dts[-1])
            states.append(W)
            dts.append(nxt)
        series = torch.stack([(X[0] + X[3] - X[6]).reshape(-1)[at] for X in states[1:]])
    off = series - tgt
    bar, bar_dt, bar_par = [torch.zeros_like(H) for _ in range(6)], torch.zeros((), dtype=torch.float64, device=dev), torch.zeros_like(par)

    def passive(n):  # gauge terms of state n, then the projection: thin layers are passive
        for k in (0, 3):
            if n:
                bar[k].view(-1).index_add_(0, at, 2.0 * off[n - 1])
            for q in range(k, k + 3):
                bar[q] = torch.where(states[n][k] < thin, torch.zeros_like(H), bar[q])

    def pull(n, f):
        nonlocal bar_par
        X = [v.detach().clone().requires_grad_() for v in states[n][:6]]
        dt = dts[n].detach().clone().requires_grad_()
        outs, bars = f(_Scheme(p, dev, par), X + [H], dt)
        pairs = [(o, b) for o, b in zip(outs, bars) if o.requires_grad]
        g = torch.autograd.grad([o for o, _ in pairs], X + [dt, par], [b for _, b in pairs], allow_unused=True)
        g = [torch.zeros_like(v) if d is None else d for d, v in zip(g, X + [dt, par])]
        bar_par = bar_par + g[7]
        return g[:6], g[6]

    def of_step(sch, X, dt):
        out, nxt = sch.step(X, dt)
        return out[:6] + [nxt], bar + [bar_dt]

    for n in range(steps, 0, -1):
        passive(n)
        bar, bar_dt = pull(n - 1, of_step)
    more, _ = pull(0, lambda sch, X, dt: ([sch.first_dt(X)], [bar_dt]))
    bar = [a.clone() + b for a, b in zip(bar, more)]
    passive(0)
    return float((off ** 2).sum()), series.cpu().numpy(), dict(zip(VARS, bar)), bar_par


def exact(case, seed):
    scenes = _scenes(case, seed)
    p, state, gauges = scenes[0]
    do = case["do"]
    if do in ("gradient", "calibration"):
        got = [_reverse(p, st, g, t, case["steps"], 0.1) for (p, st, g), t in zip(scenes, _targets(case, scenes, seed))]
        if do == "gradient":
            return {"misfit": got[0][0], "series": got[0][1], "state": got[0][2], "params": got[0][3]}
        return {"misfits": np.array([g[0] for g in got]), "series": [g[1] for g in got], "state": [g[2] for g in got],
                "params": torch.stack([g[3] for g in got])}
    if do == "ensemble":
        return [dict(zip(VARS[:6], _march(p, st, case["steps"])[0])) for p, st, _ in scenes]
    if do == "forecast":
        ends = [(k + 1) * _interval(case) for k in range(case["readings"])]
        W, t, dt, top, when, rows = _march(p, state, readings=ends, gauges=gauges)
        return {"state": torch.stack(W), "eta_max": top, "eta_time": when, "series": rows}
    W, t, dt, top, when, _ = _march(p, state, case["steps"])
    if do == "noalloc":
        return {"state": torch.stack(W), "time": t, "dt": float(dt)}
    if case.get("options"):
        return {"state": torch.stack(W), "eta_max": top, "eta_time": when}
    return {"state": torch.stack(W)}
