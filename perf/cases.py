"""Timed cases of the radiation solver, through its public entry points.

Each case is one piece of work a program using this package does: time steps
of a resident problem and the read-back of its moments, in each arithmetic
form (plain FP64, FP32 precision, fast FP64) and streaming type; a restart from
and to a host state; tables rebuilt before every step; a batch of uneven
problems; the adjoint of a run; and a whole run from its inputs.  Grids range
from the 100 x 100 beam to the 400 x 400 x 64 scattering problem of the
benchmark, with odd and ragged sizes among them.

A case is a dict of plain values:
  kind    steps, restart, tables, batch, adjoint or run
  scene   beam, shell, scatter or moving (below)
  form    plain, fast64 or fp32
  flat, adaptive   the streaming type
  nx, ny, nd, nf   interior cells, directions, Fourier harmonics
  steps, tol       time steps of one pass, tolerance of the geodesic tables

Moments of the FP32 form are 32-bit values that the boundary hands out widened
to doubles; they are returned as the 32-bit values they are.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("2dradiation_b200")

FORMS = {"plain": pkg.PLAIN_FP64, "fast64": pkg.FAST_FP64, "fp32": pkg.PRECISION_FP32}
MOMENTS = ("E", "Fx", "Fy", "Pxx", "Pxy", "Pyy")


def _case(name, kind, scene, form, nx, ny, nd, nf, steps, flat=False, adaptive=False, tol=1e-10, problems=1):
    c = dict(kind=kind, scene=scene, form=form, nx=nx, ny=ny, nd=nd, nf=nf, steps=steps, flat=flat,
             adaptive=adaptive, tol=tol, problems=problems)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # one step of the smallest problem and its moments: a program that
        # looks at every step (launches and latency)
        _case("beam_one_step_fp32", "steps", "beam", "fp32", 100, 100, 20, 5, 1, flat=True),
        # the beam from its inputs to its results in one call, in the default form
        _case("beam_whole_run_plain", "run", "beam", "plain", 100, 100, 20, 5, 500, flat=True, tol=1e-4),
        # the emitting shell around a black hole, default form
        _case("shell_plain_200x32", "steps", "shell", "plain", 200, 200, 32, 5, 100),
        # the benchmark's scattering problem in the three forms
        _case("scatter_fp32_400x64", "steps", "scatter", "fp32", 400, 400, 64, 16, 200),
        _case("scatter_fast64_400x64", "steps", "scatter", "fast64", 400, 400, 64, 16, 100),
        _case("scatter_plain_400x64", "steps", "scatter", "plain", 400, 400, 64, 16, 40),
        # a checkpoint loaded, stepped and saved: a moving fluid with active
        # sources on a ragged grid and a direction count off every multiple
        _case("restart_moving_fast64", "restart", "moving", "fast64", 237, 181, 36, 5, 100),
        # the adaptive streaming types: curved in FP32, flat in the default form
        _case("adaptive_fp32_256x64", "steps", "scatter", "fp32", 256, 256, 64, 9, 40, adaptive=True),
        _case("adaptive_flat_plain", "steps", "scatter", "plain", 151, 170, 33, 5, 40, flat=True, adaptive=True),
        # uneven independent problems stepped together (a parameter study)
        _case("batch_fp32_16", "batch", "shell", "fp32", 256, 256, 64, 5, 64, problems=16),
        # a gradient of a fit: forward with checkpoints, then backward
        _case("adjoint_256x48", "adjoint", "shell", "plain", 256, 256, 48, 5, 40),
        # geodesic tables rebuilt before every step (the updateFourierHarmonics option)
        _case("tables_each_step_fp32", "tables", "scatter", "fp32", 400, 400, 64, 16, 4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "restart", "tables", "batch", "adjoint", "run"])
    nx, ny = _log_int(rng, 48, 400), _log_int(rng, 48, 400)
    nd = rng.choice([16, 20, 24, 32, 33, 36, 48, 50, 64])
    nf = rng.choice([5, 5, 9, 16])
    form = rng.choice(["plain", "fp32", "fp32", "fast64"])
    flat = rng.random() < 0.3
    adaptive = kind == "steps" and form != "fast64" and rng.random() < 0.3
    scene = rng.choice(["shell", "scatter", "moving"])
    problems = 1
    if kind == "batch":
        nx, ny, form, scene, problems = min(nx, 256), min(ny, 256), "fp32", "shell", rng.choice([6, 9, 12])
    if kind == "adjoint":
        nx, ny, form, scene = min(nx, 256), min(ny, 256), "plain", "shell"
    if kind == "run":
        nx, ny, scene, flat = min(nx, 128), min(ny, 128), "beam", True
    if kind == "tables":
        flat, scene = False, "scatter"
    # about a tenth to a whole of the largest listed pass
    cost = nx * ny * nd * problems * (3.0 if form != "fp32" else 1.0) * (5.0 if adaptive else 1.0)
    most = 4 if kind == "tables" else (64 if kind in ("batch", "adjoint") else 400)
    steps = max(1, min(most, int(rng.uniform(0.1, 0.5) * 2e9 / cost)))
    return _case(None, kind, scene, form, nx, ny, nd, nf, steps, flat=flat, adaptive=adaptive,
                 tol=rng.choice([1e-10, 1e-8]), problems=problems)


# --------------------------------------------------------------------- inputs
def _radiation(rng, X, Y, is_flat, n_dir):
    """A radiation field as a run leaves it: smooth, brighter near the middle,
    its flux turning around the centre; nothing inside the excision."""
    r = np.sqrt(X * X + Y * Y)
    phi = (np.arange(n_dir) + 0.5) * (2 * math.pi / n_dir)
    p = rng.uniform(0.2, 0.6, 4)
    E = (0.3 + np.exp(-r / 4.0)) * (1.0 + p[0] * np.sin(p[1] * 2 * X + 1.0) * np.cos(p[2] * 2 * Y + 0.5))
    angle = np.arctan2(Y + 0.3 * np.sin(X), X + 0.2 * np.cos(Y)) + p[3]
    width = 0.8 + 0.4 * np.sin(0.7 * X + 0.9 * Y)
    I = E[:, None] * np.exp(width[:, None] * np.cos(phi[None, :] - angle[:, None]))
    if not is_flat:
        I[r <= 2.4] = 0.0
    return I


def _problem(case, rng):
    """The dict the package's Radiation takes, and the intensities to start
    from (None: the sources only)."""
    nx, ny, nd = case["nx"], case["ny"], case["nd"]
    W = pkg.workloads
    flat, scene = case["flat"], case["scene"]
    box = 1.0 if scene == "beam" else 6.0
    stream = {(True, False): W.FLAT_FIXED, (False, False): W.CURVED_FIXED, (True, True): W.FLAT_ADAPTIVE,
              (False, True): W.CURVED_ADAPTIVE}[(flat, case["adaptive"])]
    X, Y, _, _ = W.grid_coords(nx, ny, (-box, -box), (box, box))
    n, z = X.size, np.zeros(X.size)
    f = {k: z.copy() for k in ("kappa0", "kappa1", "kappaA", "eta", "ux", "uy", "initial_E_LF", "initial_Fx_LF",
                               "initial_Fy_LF", "initial_Pxx_LF", "initial_Pxy_LF", "initial_Pyy_LF")}
    f["is_initial"], f["initial_I"] = np.zeros(n, dtype=np.uint8), np.zeros(n * nd)
    I0, r = None, np.sqrt(X * X + Y * Y)
    if scene == "beam":
        src = (np.arange(n) % (nx + 2) <= 1) & (np.abs(Y) <= 0.1)
        f["is_initial"][src] = 1
        b = rng.uniform(0.5, 1.5, int(src.sum()))
        for d in (0, nd - 1):
            f["initial_I"].reshape(n, nd)[src, d] = b
    elif scene == "shell":
        f["eta"][(r >= 3.8) & (r <= 4.2)] = 1.0
        f["kappaA"] = np.where(r < 5.0, rng.uniform(0.0, 0.5, n), 0.0)
        if case["kind"] in ("batch", "adjoint"):
            f["kappa0"] = np.where(r < 5.0, rng.uniform(0.0, 1.0, n), 0.0)
            I0 = _radiation(rng, X, Y, flat, nd)
    elif scene == "scatter":
        f["kappaA"] = np.exp(-1.0 + 0.5 * rng.standard_normal(n))
        f["kappa0"] = rng.uniform(0.0, 2.0, n)
        f["eta"] = np.exp(-((X - 3.0) ** 2 + Y ** 2) / 0.5)
        I0 = _radiation(rng, X, Y, flat, nd)
    else:
        f["kappa0"], f["kappa1"] = rng.uniform(0.0, 1.5, n), rng.uniform(0.0, 0.3, n)
        f["kappaA"] = rng.uniform(0.0, 0.5, n)
        f["eta"] = np.exp(-((X - 3.0) ** 2 + (Y + 1.0) ** 2) / 2.0)
        f["ux"], f["uy"] = rng.uniform(-0.15, 0.15, n), rng.uniform(-0.15, 0.15, n)
        I0 = _radiation(rng, X, Y, flat, nd)
        src = (np.abs(X + 4.0) < 1.0) & (np.abs(Y - 3.0) < 1.0)
        f["is_initial"][src] = 1
        f["initial_I"].reshape(n, nd)[src] = 1.5 * I0[src]
    prob = dict(name=scene, nx_=nx, ny_=ny, start=(-box, -box), end=(box, box), cfl=0.9,
                metric_kind=W.MINKOWSKI if flat else W.KERRSCHILD, m=1.0, a=0.0, excision=-1.0 if flat else 2.4,
                n_dir=nd, n_fourier=case["nf"], streaming_type=stream, initial_data_type=W.INTENSITIES,
                keep_source_nodes_active=int(scene in ("beam", "moving")), n_steps=case["steps"],
                rk_tol=case["tol"], fields=f)
    return prob, I0


def _members(case):
    """The problems of a batch: grids of a half to a whole of the case's,
    directions of a quarter to a whole, flat and curved in turn."""
    out = []
    for k in range(case["problems"]):
        m = dict(case, nx=max(16, case["nx"] * (4 - k % 3) // 4 - k % 5), ny=max(16, case["ny"] * (2 + k % 3) // 4),
                 nd=max(8, case["nd"] // (1, 2, 4)[k % 3]), flat=k % 2 == 1)
        out.append(m)
    return out


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    return [_problem(m, rng) for m in (_members(case) if case["kind"] == "batch" else [case])]


def _dL(case, seed):
    return np.random.default_rng(seed + 77).uniform(-1.0, 1.0, (case["nx"] + 2) * (case["ny"] + 2))


# ------------------------------------------------------------------- the work
def prepare(case, seed):
    inputs = _inputs(case, seed)
    st = dict(case=case, inputs=inputs, form=FORMS[case["form"]])
    if case["kind"] == "run":
        return st
    st["rads"] = []
    for prob, I0 in inputs:
        r = pkg.prepare(prob, st["form"])
        if I0 is not None:
            r.set_intensity(I0)
        st["rads"].append(r)
    if case["kind"] == "tables":
        st["rads"][0].update_tables_each_step(True, case["tol"])
    elif case["kind"] == "batch":
        st["batch"] = pkg.Batch(st["rads"])
    elif case["kind"] == "adjoint":
        st["adjoint"], st["dL"] = pkg.Adjoint(st["rads"][0], 20), _dL(case, seed)
    return st


def _moments(case, rad):
    m = rad.moments_if()
    return {k: v.astype(np.float32) for k, v in m.items()} if case["form"] == "fp32" else m


def run(state):
    case = state["case"]
    kind, n = case["kind"], case["steps"]
    if kind == "run":
        res = pkg.run(state["inputs"][0][0], state["form"])
        keep = MOMENTS + ("I", "E_LF", "Fx_LF", "Fy_LF", "Pxx_LF", "Pxy_LF", "Pyy_LF", "F_LF")
        as_type = np.float32 if case["form"] == "fp32" else np.float64
        return {k: res[k].astype(as_type, copy=False) for k in keep}
    rad = state["rads"][0]
    if kind == "batch":
        state["batch"].step(n)
        return [np.stack([m[k] for k in MOMENTS]) for m in (_moments(case, r) for r in state["rads"])]
    if kind == "adjoint":
        state["adjoint"].forward(n)
        return {"gradient": state["adjoint"].backward(state["dL"]), "moments": rad.moments_if()}
    if kind == "restart":
        rad.set_intensity(state["inputs"][0][1])
        rad.step(n)
        I = rad.intensity()
        return {"moments": _moments(case, rad), "I": I.astype(np.float32) if case["form"] == "fp32" else I}
    rad.step(n)
    return _moments(case, rad)


def work(case):
    """Each step reads and writes the state once and reads 8 fields and writes
    6 moments per cell; arithmetic per (cell, direction): the departure's
    4 corners of 5 (curved) or 1 taps, the moments and one collide cycle."""
    size = 4 if case["form"] == "fp32" else 8
    total = {"bytes": 0.0, "flops": 0.0}
    for m in _members(case) if case["kind"] == "batch" else [case]:
        cells, nd, n = m["nx"] * m["ny"], m["nd"], m["steps"]
        b = n * cells * size * (2.0 * nd + 14.0) + 6 * 8 * cells
        per = (10.0 if m["flat"] else 50.0) + 12.0 + 24.0
        if m["adaptive"]:
            per += 4 * 30.0 + (0.0 if m["flat"] else 12.0 * m["nf"])
        fl = n * cells * nd * per
        if case["kind"] == "restart":
            b += 2 * 8.0 * cells * nd
        elif case["kind"] == "tables":  # about 8 trials of 6 stages of 450 operations per geodesic
            b += n * cells * 5 * 8.0 * m["nf"]
            fl += n * cells * (m["nf"] * 8 * 6 * 450.0 + 10.0 * m["nf"] ** 2 + 10.0 * m["nf"] * nd)
        elif case["kind"] == "adjoint":  # the forward's states again, the adjoint state in 32 bits
            b += n * cells * nd * (8.0 + 2 * 4.0)
            fl += 2 * fl
        total["bytes"] += b
        total["flops"] += fl
    return total


# ------------------------------------------- the same numbers in 64-bit torch
_PI = math.pi


def _sin(x):
    """The method's polynomial sine (the stencil's directions are its values)."""
    x = torch.where(x <= _PI / 2, x, torch.where(x <= 3 * _PI / 2, -(x - _PI), x - 2 * _PI)) * (2.0 / _PI)
    q = x * x
    return x * (1.57079631847 + q * (-0.64596371106 + q * (0.07968967928 + q * (-0.00467376557 + q * 0.00015148419))))


def _cos(x):
    """The method's cosine: single-precision argument and result."""
    x = x.float()
    pi, half = torch.tensor(_PI).float().to(x.device), torch.tensor(_PI / 2).float().to(x.device)
    v = torch.where(x >= pi, -_sin((x - half).double()), _sin((x + half).double()))
    return v.float().double()


def _phi(x, y):
    """The method's polynomial angle in [0, 2 pi)."""
    def atan(z):
        q = z * z
        return z * (0.9998660 + q * (-0.3302995 + q * (0.1801410 + q * (-0.0851330 + q * 0.0208351))))
    steep = x.abs().float() <= y.abs().float()
    a = atan(torch.where(steep, torch.where(y == 0, 0.0, x / torch.where(y == 0, 1.0, y)),
                         y / torch.where(x == 0, 1.0, x)))
    p = torch.where(steep, torch.where(y > 0, -a + _PI / 2, -a - _PI / 2),
                    torch.where(x > 0, a, torch.where(y >= 0, a + _PI, a - _PI)))
    p = torch.where((x == 0) & (y == 0), torch.zeros_like(p), p)
    return torch.where(p < 0, p + 2 * _PI, p)


class _Exact:
    """One problem: the method's grid, stencil, metric, tables and step."""

    def __init__(self, prob, device):
        self.prob, self.dev = prob, device
        nx_, ny_ = prob["nx_"], prob["ny_"]
        self.nx, self.ny, self.nd, self.nf = nx_ + 2, ny_ + 2, prob["n_dir"], prob["n_fourier"]
        (sx, sy), (ex, ey) = prob["start"], prob["end"]
        self.dx, self.dy = (ex - sx) / (nx_ - 1.0), (ey - sy) / (ny_ - 1.0)
        self.sx, self.sy, self.ex, self.ey = sx - self.dx, sy - self.dy, ex + self.dx, ey + self.dy
        self.dt = prob["cfl"] * min(self.dx, self.dy)
        t = self.t
        self.X = (self.sx + t(range(self.nx)) * self.dx)[None, :].expand(self.ny, self.nx).reshape(-1)
        self.Y = (self.sy + t(range(self.ny)) * self.dy)[:, None].expand(self.ny, self.nx).reshape(-1)
        n = torch.arange(self.nx * self.ny, device=device)
        i, j = n % self.nx, n // self.nx
        self.inner = n[(i > 0) & (i < self.nx - 1) & (j > 0) & (j < self.ny - 1)]
        self.curved = prob["metric_kind"] != pkg.MINKOWSKI
        self.adaptive = prob["streaming_type"] in (pkg.FLAT_ADAPTIVE, pkg.CURVED_ADAPTIVE)
        self.ex2 = (prob["excision"] * prob["m"]) ** 2 if self.curved else -1.0
        self.hole = (self.X ** 2 + self.Y ** 2 <= self.ex2)
        self.phi = 2 * _PI * (t(range(self.nd)) + 0.5) / self.nd
        self.cx, self.cy = _cos(self.phi), _sin(self.phi)
        self.rows()
        self.fixed = None
        self.alpha = torch.ones_like(self.X)
        if self.curved:
            self.metric()
            self.tables()
        self.fields()

    def t(self, v):
        return torch.as_tensor(np.asarray(v, dtype=np.float64), device=self.dev)

    def rows(self):
        """The angular interpolation's rows: 10 per direction, cubic through
        the 4 directions around the row's angle."""
        nd, ng = self.nd, 10 * self.nd
        phi = self.phi.cpu().numpy()
        g = 2 * _PI * np.arange(ng) / ng
        delta = np.abs(g[:, None] - phi[None, :])
        near = np.argmin(np.minimum(delta, 2 * _PI - delta), axis=1)
        left = np.fmod(phi[near] + _PI - g, 2 * _PI) < _PI
        idx = (near[:, None] + np.where(left, -1, -2)[:, None] + np.arange(4)[None, :] + nd) % nd
        p = np.fmod(phi[idx] + _PI - g[:, None] + 2 * _PI, 2 * _PI)
        w = np.ones((ng, 4))
        for a in range(4):
            for b in range(4):
                if a != b:
                    w[:, a] *= (_PI - p[:, b]) / (p[:, a] - p[:, b])
        self.ng, self.ig, self.igw = ng, torch.as_tensor(idx, device=self.dev), self.t(w)

    def g_lower(self, x, y):
        m = self.prob["m"]
        r2 = x * x + y * y
        r2 = torch.where(r2 > 0, r2, torch.ones_like(r2))
        r = torch.sqrt(r2)
        H = torch.where((x == 0) & (y == 0), torch.zeros_like(r), m / r)
        l = (torch.ones_like(x), r * x / r2, r * y / r2)
        return {(a, b): (-1.0 if a == b == 0 else float(a == b)) + 2 * H * l[a] * l[b]
                for a in range(3) for b in range(a, 3)}

    @staticmethod
    def inverse(g):
        # the order of the products is the method's: its differences of step
        # 1e-8 are taken of these numbers, rounding and all
        a = g[1, 1] * g[2, 2] - g[1, 2] * g[1, 2]
        b = g[1, 2] * g[0, 2] - g[0, 1] * g[2, 2]
        c = g[0, 1] * g[1, 2] - g[1, 1] * g[0, 2]
        v = 1.0 / (g[0, 0] * a + g[0, 1] * b + g[0, 2] * c)
        return {(0, 0): a * v, (0, 1): (g[0, 2] * g[1, 2] - g[0, 1] * g[2, 2]) * v,
                (0, 2): (g[0, 1] * g[1, 2] - g[0, 2] * g[1, 1]) * v, (1, 1): (g[0, 0] * g[2, 2] - g[0, 2] * g[0, 2]) * v,
                (1, 2): (g[0, 2] * g[0, 1] - g[0, 0] * g[1, 2]) * v, (2, 2): (g[0, 0] * g[1, 1] - g[0, 1] * g[0, 1]) * v}

    def metric(self):
        """The node fields that the geodesics read: lapse, shift, curvature,
        3-metric and their derivatives (4th-order differences of step 1e-8)."""
        x, y, h = self.X, self.Y, 1e-8
        low = self.g_lower(x, y)
        up = self.inverse(low)

        def deriv(ax, ay, f):
            p = [f(self.g_lower(x + k * h * ax, y + k * h * ay)) for k in (-2, -1, 1, 2)]
            return {k: (1 / 12.0 * p[0][k] - 1 / 12.0 * p[3][k] - 2 / 3.0 * p[1][k] + 2 / 3.0 * p[2][k]) / h
                    for k in p[0]}
        dl = [None, deriv(1, 0, lambda g: g), deriv(0, 1, lambda g: g)]
        du = [None, deriv(1, 0, self.inverse), deriv(0, 1, self.inverse)]
        al = 1.0 / torch.sqrt(-up[0, 0])
        b = [None, al * al * up[0, 1], al * al * up[0, 2]]
        gu = {(p, q): up[p, q] + b[p] * b[q] / (al * al) for p, q in ((1, 1), (1, 2), (2, 2))}
        da = [None] + [du[k][0, 0] / (2.0 * (-up[0, 0]) ** 1.5) for k in (1, 2)]
        db = {(k, c): al * al * du[k][0, c] + 2.0 * up[0, c] * al * da[k] for k in (1, 2) for c in (1, 2)}
        key = lambda p, q: (min(p, q), max(p, q))  # noqa: E731
        K = {}
        for p, q in ((1, 1), (1, 2), (2, 2)):
            K[p, q] = sum(2.0 * low[key(p, c)] * db[q, c] + dl[c][key(p, q)] * b[c] for c in (1, 2)) / (2.0 * al)
        s = 1.0 / torch.sqrt(gu[1, 1])
        t11, t21, t22 = 1.0 / s, s * gu[1, 2], 1.0 / torch.sqrt(low[2, 2])
        self.alpha, self.tet = al, (t11, t21, t22)
        # the tetrad's inverse: a lower triangular block
        i11, i22, i21 = 1.0 / t11, 1.0 / t22, -t21 / (t11 * t22)
        names = [al, b[1], b[2], da[1], da[2], db[1, 1], db[1, 2], db[2, 1], db[2, 2], K[1, 1], K[1, 2], K[2, 2],
                 gu[1, 1], gu[1, 2], gu[2, 2], dl[1][1, 1], dl[1][1, 2], dl[1][2, 2], dl[2][1, 1], dl[2][1, 2],
                 dl[2][2, 2], t11, t21, t22, i11, i21, i22]
        self.nodes = torch.stack(names)
        flat = torch.zeros(len(names), dtype=torch.float64, device=self.dev)
        flat[[0, 12, 14, 21, 23, 24, 26]] = 1.0
        self.outside_value = flat

    def outside(self, x, y):
        return (x > self.ex) | (x < self.sx) | (y > self.ey) | (y < self.sy)

    def at(self, x, y, first, last):
        """Node fields [first, last) at points, bilinear; flat space outside."""
        fi, fj = (x - self.sx) / self.dx, (y - self.sy) / self.dy
        i = fi.floor().clamp(0, self.nx - 2).long()
        j = fj.floor().clamp(0, self.ny - 2).long()
        tx, ty, n = fi - i, fj - j, i + j * self.nx
        f = self.nodes[first:last]
        v = (f[:, n] * (1 - tx) + f[:, n + 1] * tx) * (1 - ty) + (f[:, n + self.nx] * (1 - tx) + f[:, n + self.nx + 1] * tx) * ty
        return torch.where(self.outside(x, y), self.outside_value[first:last, None], v)

    def rhs(self, s):
        x, y, v1, v2, nu = s
        L = self.at(x, y, 0, 21)
        al, b, da = L[0], (None, L[1], L[2]), (None, L[3], L[4])
        db = {(1, 1): L[5], (1, 2): L[6], (2, 1): L[7], (2, 2): L[8]}
        K = {(1, 1): L[9], (1, 2): L[10], (2, 1): L[10], (2, 2): L[11]}
        gu = {(1, 1): L[12], (1, 2): L[13], (2, 1): L[13], (2, 2): L[14]}
        dg = {(k, p, q): L[15 + 3 * (k - 1) + p + q - 2] for k in (1, 2) for p in (1, 2) for q in (1, 2)}
        v = (None, v1, v2)
        R = (1, 2)
        Kvv = sum(K[i, j] * v[i] * v[j] for i in R for j in R)
        vda = v1 * da[1] + v2 * da[2]
        dv = []
        for k in R:
            a = v[k] * vda - al * v[k] * Kvv
            for i in R:
                a = a - gu[k, i] * da[i] - v[i] * db[i, k] + 2.0 * al * gu[i, k] * sum(K[i, j] * v[j] for j in R)
                for j in R:
                    for l in R:
                        a = a - al * 0.5 * gu[k, l] * (dg[i, l, j] + dg[j, i, l] - dg[l, i, j]) * v[i] * v[j]
            dv.append(a)
        return torch.stack([al * v1 - b[1], al * v2 - b[2], dv[0], dv[1], (al * Kvv - vda) * nu])

    def tables(self):
        """Backtraces over dt (Runge-Kutta-Fehlberg with the method's
        coefficients and step control) and their Fourier coefficients."""
        n, nf = self.inner, self.nf
        ph = 2 * _PI * (self.t(range(nf)) + 0.5) / nf
        x, y = self.X[n].repeat_interleave(nf), self.Y[n].repeat_interleave(nf)
        c1, c2 = _cos(ph).repeat(n.numel()), _sin(ph).repeat(n.numel())
        t11, t21, t22 = self.at(x, y, 21, 24)
        s = torch.stack([x, y, t11 * c1, t21 * c1 + t22 * c2, torch.ones_like(x)])
        bh = self.hole[n].repeat_interleave(nf)
        s[2:4, bh] = 0.0
        left, h = torch.full_like(x, self.dt), torch.full_like(x, self.dt)
        live, tol = (~bh).nonzero()[:, 0], self.prob["rk_tol"]
        A = ((1 / 4,), (3 / 32, 9 / 32), (1932 / 2197, -7200 / 2197, 7296 / 2197),
             (439 / 216, -8, 3680 / 513, -845 / 4104), (-8 / 27, 2, -3544 / 2565, 1859 / 4104, -11 / 44))
        B = (16 / 135, 0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55)
        T = (1 / 360, 0, -128 / 4275, -2197 / 75240, 1 / 50, 2 / 55)
        for _ in range(100000):
            if not live.numel():
                break
            y0, hh = s[:, live], torch.minimum(h[live], left[live])
            k = [self.rhs(y0)]
            for row in A:
                k.append(self.rhs(y0 - hh * sum(a * q for a, q in zip(row, k) if a)))
            e = sum(a * q[2:4] for a, q in zip(T, k) if a) * hh
            te = torch.sqrt(e[0] ** 2 + e[1] ** 2)
            ok = te <= tol
            new = torch.where(ok, y0 - hh * sum(a * q for a, q in zip(B, k) if a), y0)
            s[:, live] = new
            left[live] = torch.where(ok, left[live] - hh, left[live])
            h[live] = hh * 0.95 * (tol / (te + 1e-50)) ** 0.25
            gone = ok & ((new[0] ** 2 + new[1] ** 2 <= self.ex2) | self.outside(new[0], new[1]))
            live = live[~gone & (left[live] > 1e-14 * self.dt)]
        i11, i21, i22 = self.at(s[0], s[1], 24, 27)
        data = torch.stack([1.0 / s[4], s[0], s[1], i11 * s[2], i21 * s[2] + i22 * s[3]]).reshape(5, -1, nf)
        data[:, self.hole[n]] = 0.0  # not read
        b = [torch.ones_like(ph)]
        for k in range(1, nf):
            b.append(math.sqrt(2) * (torch.cos(ph * (k + 1) / 2) if k % 2 else torch.sin(ph * k / 2)))
        self.coef = data @ torch.stack(b, -1) / nf

    def fields(self):
        f, n = self.prob["fields"], self.inner
        q = {k: self.t(f[k])[n] for k in ("kappa0", "kappa1", "kappaA", "eta", "ux", "uy")}
        t11, t21, t22 = [v[n] for v in self.tet] if self.curved else (1.0, 0.0, 1.0)
        self.u1, self.u2 = t11 * q["ux"], t21 * q["ux"] + t22 * q["uy"]
        self.lor = 1.0 / torch.sqrt(1.0 - self.u1 ** 2 - self.u2 ** 2)
        self.adt = self.alpha[n] * self.dt
        self.eta, self.k0, self.k3, self.ka = q["eta"], q["kappa0"], 3 * q["kappa1"], q["kappaA"]
        src = torch.as_tensor(np.asarray(f["is_initial"]), device=self.dev).nonzero()[:, 0]
        self.src, self.src_I = src, self.t(f["initial_I"]).reshape(-1, self.nd)[src].T

    def corners(self, xd, yd):
        it, jt = (xd - self.sx) / self.dx, (yd - self.sy) / self.dy
        i = torch.nan_to_num(it).floor().clamp(0, self.nx - 2).long()
        j = torch.nan_to_num(jt).floor().clamp(0, self.ny - 2).long()
        fx, fy, n = it - i, jt - j, i + j * self.nx
        return [(n, (1 - fx) * (1 - fy)), (n + 1, fx * (1 - fy)), (n + self.nx, (1 - fx) * fy), (n + self.nx + 1, fx * fy)]

    def angular(self, I, n, z):
        z = torch.nan_to_num(z).clamp(1e-8, self.ng - 1e-8)
        g = z.floor().long()
        t, g1, v = z - g, (g + 1) % self.ng, 0.0
        for k in range(4):
            v = v + (1 - t) * self.igw[g, k] * I[self.ig[g, k], n] + t * self.igw[g1, k] * I[self.ig[g1, k], n]
        return v.clamp(min=0.0)

    def departures(self, new):
        """Per (direction, cell): the corners and their weights, the velocity
        at the departure, and the factor of the streamed value."""
        n = self.inner
        c1, c2 = self.cx[:, None].expand(self.nd, n.numel()), self.cy[:, None].expand(self.nd, n.numel())
        if self.adaptive:
            sn, cs = _sin(new[n]), _cos(new[n])
            c1, c2 = c1 * cs - c2 * sn, c1 * sn + c2 * cs
        if not self.curved:
            return self.corners(self.X[n] - c1 * self.dt, self.Y[n] - c2 * self.dt), c1, c2, torch.ones_like(c1)
        ph = _phi(c1, c2) if self.adaptive else self.phi[:, None].expand(c1.shape)
        f = [0.0] * 5
        for k in range(self.nf):
            b = 1.0 if k == 0 else math.sqrt(2) * (torch.cos(ph * (k + 1) / 2) if k % 2 else torch.sin(ph * k / 2))
            f = [f[q] + self.coef[q, :, k] * b for q in range(5)]
        s, xd, yd, v1, v2 = (torch.as_tensor(v).expand(c1.shape) for v in f)
        gone = self.hole[n] | (xd ** 2 + yd ** 2 <= self.ex2)
        return self.corners(xd, yd), v1, v2, torch.where(gone, torch.zeros_like(s), s ** 3 * self.alpha[n] ** 3)

    def stream(self, I, old=None, new=None):
        """Streamed values [nd, cells]; old, new: the nodes' rotation angles
        (adaptive streaming)."""
        if self.adaptive or self.fixed is None:
            corners, v1, v2, scale = self.departures(new)
            if not self.adaptive:
                z = self.ng * _phi(v1, v2) / (2 * _PI) if self.curved else None
                self.fixed = (corners, z, scale)
        if not self.adaptive:
            corners, z, scale = self.fixed
        if self.curved:
            I = I / self.alpha ** 3
        val = 0.0
        for m, w in corners:
            if self.adaptive:
                th = torch.remainder(2 * _PI - old, 2 * _PI)
                sn, cs = _sin(th)[m], _cos(th)[m]
                z = self.ng * _phi(v1 * cs - v2 * sn, v1 * sn + v2 * cs) / (2 * _PI)
            if z is None:
                val = val + w * torch.gather(I, 1, m)
            else:
                val = val + w * self.angular(I, m, z)
        return torch.where(scale == 0, torch.zeros_like(scale), scale * val)

    def collide(self, S, new=None):
        """The collided intensities and their moments (lambda iteration to
        a relative change of 1e-4 of the six moments)."""
        n1, n2 = self.cx[:, None], self.cy[:, None]
        if self.adaptive:
            sn, cs = _sin(new[self.inner]), _cos(new[self.inner])
            n1, n2 = n1 * cs - n2 * sn, n1 * sn + n2 * cs
        u1, u2, L, adt, w = self.u1, self.u2, self.lor, self.adt, 1.0 / self.nd
        un = u1 * n1 + u2 * n2
        A = L * (1.0 - un)
        sc = (1 - L * un / (L + 1)) * L
        q1, q2 = (n1 - sc * u1) / A, (n2 - sc * u2) / A
        g = 1.0 / (1.0 + adt * (self.ka + self.k0) * A)
        h = adt / (A * A) * g

        def moments(v):
            return torch.stack([(w * v * f).sum(0) for f in (1.0, n1, n2, n1 * n1, n1 * n2, n2 * n2)])
        m0 = m = moments(S)
        MA, MB, MC, MD = moments(g * S), moments(h + 0 * n1), moments(h * q1), moments(h * q2)
        live = ~self.hole[self.inner]
        F = torch.zeros_like(m[:3])
        more = live.clone()
        for _ in range(100):
            E, Fx, Fy, Pxx, Pxy, Pyy = m
            uF, ux, uy = u1 * Fx + u2 * Fy, u1 * Pxx + u2 * Pxy, u1 * Pxy + u2 * Pyy
            uu = u1 * ux + u2 * uy
            rr = L / (1.0 + L) * ((2 * L + 1.0) * uF - L * uu)
            f = torch.stack([L * L * (E - 2 * uF + uu), L * L * (Fx - L * E * u1 - ux + u1 * rr),
                             L * L * (Fy - L * E * u2 - uy + u2 * rr)])
            new_m = MA + (self.eta + self.k0 * f[0]) * MB + self.k3 * (f[1] * MC + f[2] * MD)
            with torch.no_grad():
                diff = torch.sqrt((((m - new_m) / new_m) ** 2).sum(0))
            F, m = torch.where(more, f, F), torch.where(more, new_m, m)
            more = more & (diff > 1e-4)
            if not bool(more.any()):
                break
        I = g * S + h * (self.eta + self.k0 * F[0] + self.k3 * (q1 * F[1] + q2 * F[2]))
        return torch.where(live, I, S), torch.where(live, m, m0)

    def sources(self, I):
        if self.src.numel():
            I = I.clone()
            I[:, self.src] = self.src_I
        return I

    def steps(self, I, count):
        """count steps from I [nd, nodes]; the last state and its moments."""
        mom = torch.zeros(6, self.nx * self.ny, dtype=torch.float64, device=self.dev)
        old = torch.zeros_like(self.X)
        for _ in range(count):
            if self.prob["keep_source_nodes_active"]:
                I = self.sources(I)
            new = None
            if self.adaptive:
                new = old.clone()
                fl = mom[1:3].reshape(2, self.ny, self.nx)
                avg = torch.nn.functional.avg_pool2d(fl[None], 3, 1)[0].reshape(2, -1)
                E, norm = mom[0, self.inner], torch.sqrt((avg ** 2).sum(0))
                turn = (E > 1e-16) & (norm > 0.01 * E)
                new[self.inner] = torch.where(turn, _phi(avg[0], avg[1]), old[self.inner])
            v, m = self.collide(self.stream(I, old, new), new)
            I = I.index_copy(1, self.inner, v)
            mom = torch.zeros_like(mom).index_copy(1, self.inner, m)
            old = new if self.adaptive else old
        return I, mom

    def lab_moments(self, mom):
        """Lab-frame moments (flat space: the same tensor) and |F|."""
        E, Fx, Fy, Pxx, Pxy, Pyy = mom
        return dict(zip(("E_LF", "Fx_LF", "Fy_LF", "Pxx_LF", "Pxy_LF", "Pyy_LF", "F_LF"),
                        (E, Fx, Fy, Pxx, Pxy, Pyy, torch.sqrt(Fx ** 2 + Fy ** 2))))


def exact(case, seed):
    gpu = torch.cuda.is_available()
    members = _members(case) if case["kind"] == "batch" else [case]
    size = sum(m["nx"] * m["ny"] * m["nd"] * m["steps"] * (4 if m["adaptive"] else 1) for m in members)
    if size * (4 if case["kind"] == "adjoint" else 1) > (8e9 if gpu else 3e7):  # about 20 seconds
        return None
    device, out = torch.device("cuda" if gpu else "cpu"), []
    for prob, I0 in _inputs(case, seed):
        p = _Exact(prob, device)
        nodes = p.nx * p.ny
        I = p.t(I0).reshape(nodes, p.nd).T if I0 is not None else torch.zeros(p.nd, nodes, dtype=torch.float64, device=device)
        if I0 is None:
            I = p.sources(I)
        if case["kind"] == "adjoint":
            out.append(_exact_adjoint(p, I, case, seed))
            continue
        I, mom = p.steps(I, prob["n_steps"])
        if case["kind"] == "batch":
            out.append(mom.cpu().numpy())
            continue
        m = {k: v.cpu().numpy() for k, v in zip(MOMENTS, mom)}
        if case["kind"] == "run":
            m.update(I=I.T.reshape(-1).cpu().numpy(), **{k: v.cpu().numpy() for k, v in p.lab_moments(mom).items()})
        elif case["kind"] == "restart":
            m = {"moments": m, "I": I.T.reshape(-1).cpu().numpy()}
        out.append(m)
    return out if case["kind"] == "batch" else out[0]


def _exact_adjoint(p, I, case, seed):
    """Gradients by automatic differentiation, one step recomputed at a time."""
    states, mom = [], None
    with torch.no_grad():
        for _ in range(case["steps"]):
            states.append(I)
            I, mom = p.steps(I, 1)
    dL = p.t(_dL(case, seed))
    names = {"eta": "eta", "kappaA": "ka", "kappa0": "k0"}
    grad = {k: torch.zeros(p.nx * p.ny, dtype=torch.float64, device=p.dev) for k in names}
    lam = None
    for I0 in reversed(states):
        I0 = I0.detach().requires_grad_(True)
        for a in names.values():
            setattr(p, a, getattr(p, a).detach().requires_grad_(True))
        I1, m = p.steps(I0, 1)
        # the loss reads E of the last state at colliding cells
        if lam is None:
            live = (~p.hole[p.inner]).double()
            loss = (dL[p.inner] * live * I1[:, p.inner].sum(0) / p.nd).sum()
        else:
            loss = (lam * I1).sum()
        g = torch.autograd.grad(loss, [I0] + [getattr(p, a) for a in names.values()])
        # the halo is not stepped: nothing goes back through it
        lam = torch.zeros_like(g[0]).index_copy(1, p.inner, g[0][:, p.inner])
        for k, v in zip(names, g[1:]):
            grad[k][p.inner] += v
    return {"gradient": {k: v.cpu().numpy() for k, v in grad.items()},
            "moments": {k: v.cpu().numpy() for k, v in zip(MOMENTS, mom)}}
