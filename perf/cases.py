"""The work that users of this framework have it do, as cases to be timed.

Every case goes through the public Python entry points (``api.Solver`` for
one grid, ``batch.Batch`` for many) over the C ABI.  The grid sizes, physics
and initial conditions are those of the repository's workloads (2-D MHD 256^2
turbulence, 3-D MHD 256^3 blast, 3-D RMHD 192^3 at Lorentz factors up to 10,
ensembles of 2-D MHD grids of 64 to 512 cells a side, serving mixes of MHD and
HD grids) with odd and ragged extents among them.

A single-grid pass is ``api == "step"``: one AdvanceStep whose dt is the one
the step before returned (a driver's loop), or ``api == "run"``: ``steps``
steps with the dt sequence kept on the device.  The state goes on from pass
to pass; the outputs are the whole device state and the next dt.

``exact`` restates the ideal-MHD and HD step in plain float64 torch (PLM or
PPM, HLLD/HLLC, UCT_HLLD/UCT_HLL, RK2/RK3, periodic).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from gpluto_dev_b200 import api, batch, ics

PHYSICS = {"hd": api.HD, "mhd": api.MHD, "rmhd": api.RMHD}
GAMMA = {"hd": 5.0 / 3.0, "mhd": 5.0 / 3.0, "rmhd": 4.0 / 3.0}


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def _grid(name, physics, n, precision="fp64", api_="run", steps=1, ic="turbulence", limiter="mc",
          rk=2, sides="periodic"):
    c = {"kind": "grid", "physics": physics, "ndim": len(n), "nx": n[0], "ny": n[1],
         "nz": n[2] if len(n) == 3 else 1, "precision": precision, "api": api_, "steps": steps,
         "ic": ic, "limiter": limiter, "rk": rk, "sides": sides}
    if name:
        c["name"] = name
    return c


def _batch(name, kind, grids, lo, hi, steps, layout):
    c = {"kind": kind, "grids": grids, "lo": lo, "hi": hi, "steps": steps, "layout": layout}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest grid of the ensembles on its own, stepped by a driver that reads dt back
        _grid("mhd2d-64-step", "mhd", (64, 64), api_="step"),
        # 2-D turbulence run: ten steps between a driver's looks at the state
        _grid("mhd2d-256-run", "mhd", (256, 256), steps=10),
        # the same in the mixed form on an odd grid
        _grid("mhd2d-333x171-mixed", "mhd", (333, 171), "mixed", steps=10),
        # the 3-D blast of the benchmark, a step at a time, in both forms
        _grid("mhd3d-256-blast", "mhd", (256, 256, 256), api_="step", ic="blast"),
        _grid("mhd3d-256-blast-mixed", "mhd", (256, 256, 256), "mixed", api_="step", ic="blast"),
        # a small 3-D run with no even extent
        _grid("mhd3d-61x47x53-run", "mhd", (61, 47, 53), steps=5),
        # higher-order reconstruction and RK3
        _grid("mhd3d-128x96x112-ppm-rk3", "mhd", (128, 96, 112), limiter="ppm", rk=3),
        # relativistic MHD: the 192^3 run, and a smaller one in the mixed form
        _grid("rmhd3d-192", "rmhd", (192, 192, 192), ic="jet"),
        _grid("rmhd3d-90x72x60-mixed", "rmhd", (90, 72, 60), "mixed"),
        # hydrodynamics
        _grid("hd3d-160", "hd", (160, 160, 160), steps=2),
        # open and mirrored sides, the state brought back for output every ten steps
        _grid("mhd3d-96x64x80-outflow", "mhd", (96, 64, 80), steps=10, limiter="vl",
              sides="outflow"),
        # an ensemble of uneven 2-D MHD grids, half of them mixed, twelve due for output a pass
        _batch("ensemble-128", "ensemble", 128, 64, 512, 25, 1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, ndim, lo, hi):
    """Extents of one grid: a size, and each side within a factor of 1.5 of it."""
    side = _log(rng, 1.5 * lo, hi / 1.5)
    return tuple(_log(rng, side / 1.5, side * 1.5) for _ in range(ndim))


def draw(rng: random.Random):
    what = rng.choice(["mhd2d", "mhd2d", "mhd3d", "mhd3d", "mhd3d", "rmhd3d", "hd", "sides",
                       "batch"])
    precision = rng.choice(["fp64", "mixed"])
    how = rng.choice([("step", 1), ("run", 1), ("run", rng.randint(2, 10))])
    if what == "mhd2d":
        return _grid(None, "mhd", _box(rng, 2, 48, 1024), precision, how[0], how[1],
                     limiter=rng.choice(["mc", "mc", "vl", "ppm"]), rk=rng.choice([2, 2, 3]))
    if what == "mhd3d":
        n = _box(rng, 3, 32, 256)
        return _grid(None, "mhd", n, precision, how[0], 1 if n[0] * n[1] * n[2] > 2e6 else how[1],
                     rng.choice(["blast", "turbulence"]), rng.choice(["mc", "mc", "vl", "ppm"]),
                     rng.choice([2, 2, 3]))
    if what == "rmhd3d":
        return _grid(None, "rmhd", _box(rng, 3, 48, 180), precision, how[0], 1)
    if what == "hd":
        return _grid(None, "hd", _box(rng, rng.choice([2, 3]), 32, 192), precision, how[0],
                     how[1], limiter=rng.choice(["mc", "vl"]))
    if what == "sides":
        return _grid(None, "mhd", _box(rng, 3, 32, 112), precision, "run", rng.randint(5, 10),
                     limiter=rng.choice(["mc", "vl"]), sides=rng.choice(["outflow", "mirror"]))
    kind = rng.choice(["ensemble", "serving"])
    hi = rng.randint(128, 400) if kind == "ensemble" else rng.randint(40, 72)
    return _batch(None, kind, rng.randint(16, 96), 64 if kind == "ensemble" else 24, hi,
                  rng.randint(5, 25), rng.randint(2, 1 << 20))


# ---------------------------------------------------------------------------
# Inputs: seeded random fields, made on the device
# ---------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Modes:
    """Sum of 16 cosines of integer wave vectors |k_d| <= 3 on the unit box."""

    def __init__(self, rng, ndim):
        k = rng.integers(-3, 4, size=(16, 3))
        k[:, ndim:] = 0
        k[(k == 0).all(axis=1), 0] = 1
        self.k, self.a = k, rng.uniform(0.2, 1.0, 16)
        self.p = rng.uniform(0.0, 2.0 * math.pi, 16)

    def __call__(self, n, shift, deriv=None):
        nx, ny, nz = n
        ax = [(torch.arange(m, dtype=torch.float64, device=_device()) + s) / m
              for m, s in zip(n, shift)]
        out = torch.zeros((nz, ny, nx), dtype=torch.float64, device=_device())
        for k, a, p in zip(self.k, self.a, self.p):
            th = (2.0 * math.pi * int(k[2]) * ax[2])[:, None, None] \
                + (2.0 * math.pi * int(k[1]) * ax[1])[None, :, None] \
                + (2.0 * math.pi * int(k[0]) * ax[0] + float(p))[None, None, :]
            if deriv is None:
                out += float(a) * torch.cos(th)
            else:
                out -= float(a) * 2.0 * math.pi * int(k[deriv]) * torch.sin(th)
        return out


def _up(x, d):            # value of the next cell along direction d (0 = x)
    return torch.roll(x, -1, dims=x.dim() - 1 - d)


def _dn(x, d):            # value of the previous cell along direction d
    return torch.roll(x, 1, dims=x.dim() - 1 - d)


def _inputs(physics, ndim, n, ic, seed):
    """(V [nvar, nz, ny, nx], Bs) on the device: cell primitives and left-face fields."""
    rng = np.random.default_rng([seed, ndim, *n])
    nv = 5 if physics == "hd" else 8
    c = (0.5,) * ndim + (0.0,) * (3 - ndim)
    nx, ny, nz = n
    V = torch.zeros((nv, nz, ny, nx), dtype=torch.float64, device=_device())
    f = _Modes(rng, ndim)(n, c)
    f = f / f.abs().max()
    if physics == "rmhd":
        # Lorentz factors log-uniform in [1, 10] ("jet") or [1, 2], along one bulk direction;
        # magnetisation 1
        top = math.log(10.0 if ic == "jet" else 2.0)
        V[0], V[7] = 1.0 + 0.5 * f, 0.1
        m = _Modes(rng, ndim)(n, c).reshape(-1)
        q = torch.empty_like(m)
        q[torch.argsort(m)] = (torch.arange(m.numel(), dtype=torch.float64,
                                            device=m.device) + 0.5) / m.numel()
        v = torch.sqrt(1.0 - torch.exp(-2.0 * q * top)).reshape(nz, ny, nx)
        e = rng.normal(size=3)
        e /= np.linalg.norm(e)
        for d in range(3):
            V[1 + d] = v * float(e[d])
        b2 = 1.0 * (V[0] * (1.0 + 4.0 * V[7] / V[0])).mean()
    else:
        psi = [_Modes(rng, ndim) for _ in range(3)]
        if ndim == 3:
            vel = [psi[2](n, c, 1) - psi[1](n, c, 2), psi[0](n, c, 2) - psi[2](n, c, 0),
                   psi[1](n, c, 0) - psi[0](n, c, 1)]
        else:
            vel = [psi[2](n, c, 1), -psi[2](n, c, 0), torch.zeros_like(f)]
        v2 = sum(v * v for v in vel)
        if ic == "blast":     # p = 10 in a sphere of radius 0.1, beta 0.1 outside it
            x, y, z = ((torch.arange(m, dtype=torch.float64, device=f.device) + 0.5) / m - 0.5
                       for m in n)
            r2 = x[None, None, :] ** 2 + y[None, :, None] ** 2 + z[:, None, None] ** 2
            V[0] = 1.0
            V[nv - 1] = torch.where(r2 < 0.01, 10.0, 0.1)
            s = 0.1 / torch.sqrt(v2.mean())
            b2 = torch.tensor(2.0, dtype=torch.float64)
        else:                 # rms Mach number 0.5, plasma beta 2
            V[0], V[nv - 1] = 1.0 + 0.2 * f, 1.0
            s = 0.5 / torch.sqrt((v2 * V[0] / GAMMA[physics]).mean())
            b2 = torch.tensor(1.0, dtype=torch.float64)
        for d in range(3):
            V[1 + d] = vel[d] * s
    Bs = []
    if physics != "hd":
        if ic == "blast":
            e = rng.normal(size=3)
            e /= np.linalg.norm(e)
            Bs = [torch.full_like(f, math.sqrt(float(b2)) * float(e[d])) for d in range(ndim)]
        else:                 # discrete curl of a vector potential on the edges: div B = 0
            h = [1.0 / m for m in n]
            A = [_Modes(rng, ndim)(n, tuple(0.5 if (q == d and q < ndim) else 0.0
                                            for q in range(3))) for d in range(3)]
            D = lambda a, d: (_up(A[a], d) - A[a]) / h[d]
            Bs = [D(2, 1), -D(2, 0)] if ndim == 2 else \
                [D(2, 1) - D(1, 2), D(0, 2) - D(2, 0), D(1, 0) - D(0, 1)]
            m = sum((0.5 * (b + _up(b, d))) ** 2 for d, b in enumerate(Bs)).mean()
            s = torch.sqrt(b2.to(m.device) / m)
            Bs = [b * s for b in Bs]
        for d, b in enumerate(Bs):
            V[4 + d] = 0.5 * (b + _up(b, d))
    return V, Bs


def _first_dt(n, ndim, physics):
    # well inside the CFL limit of every initial condition above; NextTimeStep raises it
    return 0.05 / max(n[:ndim]) if physics != "hd" else 0.1 / max(n[:ndim])


def _shape(case):
    return (case["nx"], case["ny"], case["nz"])


def _scheme(case, physics):
    return api.Scheme(physics=PHYSICS[physics], limiter=case["limiter"],
                      riemann="hllc" if physics == "hd" else "hlld",
                      ct_emf="uct_hll" if physics == "rmhd" else "uct_hlld",
                      precision=api.MIXED if case["precision"] == "mixed" else api.FP64,
                      gamma=GAMMA[physics], cfl=0.3 if physics == "rmhd" else 0.4, rk=case["rk"])


def _members(case):
    """(physics, shape, precision) of each grid of a batch."""
    r = random.Random(case["layout"])
    out = []
    for g in range(case["grids"]):
        precision = "fp64" if (g // 2) % 2 == 0 else "mixed"
        side = _log(r, case["lo"], case["hi"])
        if case["kind"] == "ensemble":
            out.append(("mhd", (side, side if g % 2 == 0 else side // 2, 1), precision))
        else:
            side3 = r.random() < 0.5
            n = (side, side, side) if side3 else (4 * side, 4 * side, 1)
            out.append((r.choice(["mhd", "hd"]), n, precision))
    return out


def _ndim(n):
    return 3 if n[2] > 1 else 2


def _due(case):
    return list(range(min(12, case["grids"])))


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

class _View:
    """A float64 device array of the solver's state, for torch.as_tensor, which
    keeps this object: the solver lives as long as a tensor over its memory."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False),
                                         "version": 3, "strides": None, "stream": None}


def prepare(case, seed):
    if case["kind"] == "grid":
        n, ndim, physics = _shape(case), case["ndim"], case["physics"]
        V, Bs = _inputs(physics, ndim, n, case["ic"], seed)
        sides = {}
        if case["sides"] == "outflow":      # open along x and y, mirrored along z
            sides = {"outflow": 0b001111, "reflect": 0b110000}
        elif case["sides"] == "mirror":     # mirrored along y
            sides = {"reflect": 0b001100}
        s = api.Solver(ndim, n, _scheme(case, physics),
                       nghost=3 if case["limiter"] == "ppm" else 2, **sides)
        s.upload(V.cpu().numpy(), None, [b.cpu().numpy() for b in Bs])
        return {"case": case, "solver": s, "dt": _first_dt(n, ndim, physics)}
    members = _members(case)
    states = []
    for g, (physics, n, precision) in enumerate(members):
        ndim = _ndim(n)
        V, Bs = _inputs(physics, ndim, n, "turbulence", seed * 1000 + g)
        states.append((ics.PrimState(PHYSICS[physics], ndim, n, GAMMA[physics], V.cpu().numpy(),
                                     [b.cpu().numpy() for b in Bs]),
                       _scheme({"limiter": "mc", "precision": precision, "rk": 2}, physics)))
    b = batch.Batch(sum(batch.slot_bytes(*s) for s in states) + (1 << 20), len(states))
    slots = [b.add(st, sc, _first_dt(m[1], st.ndim, m[0]), 1 << 30)
             for (st, sc), m in zip(states, members)]
    return {"case": case, "batch": b, "slots": slots}


def run(state):
    case = state["case"]
    if case["kind"] != "grid":
        b = state["batch"]
        b.advance(case["steps"])
        b.wait()
        out = {"dt": np.array([b.status(s).dt for s in state["slots"]])}
        for g in _due(case):
            V, U, Bs = b.download(state["slots"][g])
            out["grid%02d" % g] = [V, U] + Bs
        return out
    s = state["solver"]
    if case["api"] == "step":
        state["dt"] = s.AdvanceStep(state["dt"]).dt_next
    else:
        state["dt"], _, _ = s.run(case["steps"], state["dt"], history=False)
    if case["sides"] != "periodic":
        V, U, Bs = s.download()
    else:
        nx, ny, nz = s.shape
        u, v, bs = s.device_pointers()
        V = torch.as_tensor(_View(s, v, (s.nvar, nz, ny, nx)), device="cuda")
        U = torch.as_tensor(_View(s, u, (s.nvar, nz, ny, nx)), device="cuda")
        Bs = [torch.as_tensor(_View(s, p, (nz, ny, nx)), device="cuda")
              for p in (bs[:s.ndim] if case["physics"] != "hd" else [])]
    return {"V": V, "U": U, "B": Bs, "dt": state["dt"]}


def _work(physics, ndim, n, rk, steps):
    cells = n[0] * n[1] * n[2]
    # the state read and written once per stage, the step's first state read by every later one
    words = 5 if physics == "hd" else 8 + ndim + (5 if physics == "rmhd" else 0)
    # a division or a root counted as one operation; per face and per cell
    face, cell = {"hd": (150, 60), "mhd": (420, 220), "rmhd": (1600, 400)}[physics]
    return (cells * steps * words * 8.0 * (3 * rk - 1), cells * steps * rk * (ndim * face + cell))


def work(case):
    if case["kind"] == "grid":
        b, f = _work(case["physics"], case["ndim"], _shape(case), case["rk"], case["steps"])
    else:
        w = [_work(p, _ndim(n), n, 2, case["steps"]) for p, n, _ in _members(case)]
        b, f = sum(x[0] for x in w), sum(x[1] for x in w)
    return {"bytes": b, "flops": float(f)}


def tolerance(case):
    mixed = case["kind"] != "grid" or case["precision"] == "mixed"
    physics = case.get("physics", "mhd")
    if physics == "rmhd":
        # the secant on the total pressure stops at 1e-5: its exit is a decision that the last
        # bits of a quartic's roots can change in single cells
        return {"rel": 1e-7, "max": 1e-4} if mixed else {"rel": 1e-11, "max": 1e-7}
    if mixed:    # FP32 fluxes; up to 5e-8 and 1.1e-6 off the float64 step after 25 steps
        return {"rel": 2e-7, "max": 5e-6}
    return {"rel": 1e-14, "max": 1e-12}   # up to 7e-16 and 1e-14 off after 25 steps


# ---------------------------------------------------------------------------
# The step in plain float64 torch
# ---------------------------------------------------------------------------

def _mc(p, m):
    s = 2.0 * torch.where(p.abs() < m.abs(), p, m)
    q = 0.5 * (m + p)
    return torch.where(p * m > 0, torch.where(q.abs() < s.abs(), q, s), torch.zeros_like(p))


def _vl(p, m):
    return torch.where(p * m > 0, 2.0 * p * m / (p + m), torch.zeros_like(p))


def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))


def _parabola(p, m):
    """Increments to the right and left face of a cell, made monotone."""
    ext = p * m >= 0
    p2 = torch.where(p.abs() >= 2 * m.abs(), -2.0 * m, p)
    m2 = torch.where((p.abs() < 2 * m.abs()) & (m.abs() >= 2 * p.abs()), -2.0 * p, m)
    z = torch.zeros_like(p)
    return torch.where(ext, z, p2), torch.where(ext, z, m2)


def _cell_edges(V, d, limiter):
    """(value at the left face, value at the right face) of every cell along d."""
    if limiter == "ppm":
        qm, qp = _dn(V, d), _up(V, d)
        f = (-qm + 7.0 * (V + qp) - _up(qp, d)) / 12.0
        f = V + _minmod(f - V, qp - V)          # constrained right face
        p, m = _parabola(f - V, _dn(f, d) - V)
        return V + m, V + p
    s = (_mc if limiter == "mc" else _vl)(_up(V, d) - V, V - _dn(V, d))
    return V - 0.5 * s, V + 0.5 * s


def _emf_edges(b, d, limiter, field):
    """The same for the edge reconstruction (the face field always takes MC with PLM)."""
    if limiter == "ppm":
        qm, qp = _dn(b, d), _up(b, d)
        fp = b + _minmod((-qm + 5.0 * b + 2.0 * qp) / 6.0 - b, qp - b)
        fm = b + _minmod((2.0 * qm + 5.0 * b - qp) / 6.0 - b, qm - b)
        p, m = _parabola(fp - b, fm - b)
        return b + m, b + p
    return _cell_edges(b, d, "mc" if field else limiter)


def _cons_mhd(v, g):
    k = 0.5 * (v[0] * (v[1] ** 2 + v[2] ** 2 + v[3] ** 2) + v[4] ** 2 + v[5] ** 2 + v[6] ** 2)
    return torch.stack([v[0], v[0] * v[1], v[0] * v[2], v[0] * v[3], v[4], v[5], v[6],
                        k + v[7] / (g - 1.0)])


def _cons_hd(v, g):
    k = 0.5 * v[0] * (v[1] ** 2 + v[2] ** 2 + v[3] ** 2)
    return torch.stack([v[0], v[0] * v[1], v[0] * v[2], v[0] * v[3], k + v[4] / (g - 1.0)])


def _flux_mhd(v, u, d):
    vn, bn = v[1 + d], v[4 + d]
    pt = v[7] + 0.5 * (v[4] ** 2 + v[5] ** 2 + v[6] ** 2)
    f = torch.empty_like(u)
    f[0] = u[1 + d]
    for q in range(3):
        f[1 + q] = u[1 + q] * vn - v[4 + q] * bn
        f[4 + q] = v[4 + q] * vn - bn * v[1 + q]
    f[7] = (u[7] + pt) * vn - bn * (v[1] * v[4] + v[2] * v[5] + v[3] * v[6])
    f[1 + d] += pt
    return f, pt


def _fast(v, d, g):
    a2 = g * v[7]
    bt2 = v[4 + (d + 1) % 3] ** 2 + v[4 + (d + 2) % 3] ** 2
    b2 = v[4 + d] ** 2 + bt2
    c = torch.sqrt(0.5 * (a2 + b2 + torch.sqrt((a2 - b2) ** 2 + 4.0 * a2 * bt2)) / v[0])
    return v[1 + d] - c, v[1 + d] + c


def _hlld(vl, vr, Bn, d, g):
    """(flux, cmax, face data of the upwind CT) of Miyoshi & Kusano's solver."""
    t, b = (d + 1) % 3, (d + 2) % 3
    ul, ur = _cons_mhd(vl, g), _cons_mhd(vr, g)
    fl, ptl = _flux_mhd(vl, ul, d)
    fr, ptr = _flux_mhd(vr, ur, d)
    (l0, l1), (r0, r1) = _fast(vl, d, g), _fast(vr, d, g)
    Sl, Sr = torch.minimum(l0, r0), torch.maximum(l1, r1)
    cmax = torch.maximum(Sl.abs(), Sr.abs())
    dl, dr = Sl - vl[1 + d], Sr - vr[1 + d]
    w = 1.0 / (dr * ur[0] - dl * ul[0])
    SM = (dr * ur[1 + d] - dl * ul[1 + d] - ptr + ptl) * w
    pts = (dr * ur[0] * ptl - dl * ul[0] * ptr
           + vl[0] * vr[0] * dr * dl * (vr[1 + d] - vl[1 + d])) * w
    Bx = (Sr * vr[4 + d] - Sl * vl[4 + d]) / (Sr - Sl)
    sgn = torch.where(Bx > 0, 1.0, -1.0).to(Bx.dtype)
    rl, rr = ul[0] * dl / (Sl - SM), ur[0] * dr / (Sr - SM)
    hll = (rl < 0) | (rr < 0)
    ql, qr = torch.sqrt(rl), torch.sqrt(rr)
    S1L, S1R = SM - Bx.abs() / ql, SM + Bx.abs() / qr
    hllc = ((S1L - Sl) < 1e-4 * (SM - Sl)) | ((S1R - Sr) > -1e-4 * (Sr - SM))
    fh = (Sl * Sr * (ur - ul) + Sr * fl - Sl * fr) / (Sr - Sl)
    uh = (Sr * ur - Sl * ul + fl - fr) / (Sr - Sl)
    S1L, S1R = torch.where(hllc, SM, S1L), torch.where(hllc, SM, S1R)
    us = []
    for v, u, S, dv, r, pt in ((vl, ul, Sl, dl, rl, ptl), (vr, ur, Sr, dr, rr, ptr)):
        k = (u[0] * dv * dv - Bx * Bx) / (u[0] * dv * (S - SM) - Bx * Bx)
        s = torch.empty_like(u)
        s[0], s[1 + d], s[4 + d] = r, r * SM, Bx
        vs, vb = {d: SM}, SM * Bx
        for q in (t, b):
            s[4 + q] = torch.where(hllc, uh[4 + q], u[4 + q] * k)
            vs[q] = v[1 + q] - Bx / (u[0] * dv) * (s[4 + q] - u[4 + q])
            s[1 + q] = r * vs[q]
            vb = vb + vs[q] * s[4 + q]
        vb0 = v[1 + d] * Bx + v[1 + t] * u[4 + t] + v[1 + b] * u[4 + b]
        s[7] = (dv * u[7] - pt * v[1 + d] + pts * SM + Bx * (vb0 - vb)) / (S - SM)
        us.append((s, vs, vb))
    (usl, vsl, vbl), (usr, vsr, vbr) = us
    ussl, ussr = usl.clone(), usr.clone()
    vb, vss = SM * Bx, {}
    for q in (t, b):
        vss[q] = (ql * vsl[q] + qr * vsr[q] + (usr[4 + q] - usl[4 + q]) * sgn) / (ql + qr)
        bq = (ql * usr[4 + q] + qr * usl[4 + q] + ql * qr * (vsr[q] - vsl[q]) * sgn) / (ql + qr)
        ussl[4 + q], ussr[4 + q] = bq, bq
        ussl[1 + q], ussr[1 + q] = rl * vss[q], rr * vss[q]
        vb = vb + vss[q] * bq
    ussl[7] = usl[7] - ql * (vbl - vb) * sgn
    ussr[7] = usr[7] + qr * (vbr - vb) * sgn
    f = torch.where(SM >= 0, fl + S1L * (ussl - usl) + Sl * (usl - ul),
                    fr + S1R * (ussr - usr) + Sr * (usr - ur))
    f = torch.where(S1R <= 0, fr + Sr * (usr - ur), f)
    f = torch.where(S1L >= 0, fl + Sl * (usl - ul), f)
    f = torch.where(hll, fh, f)
    f = torch.where(Sr <= 0, fr, f)
    f = torch.where(Sl >= 0, fl, f)
    # face data: the two face EMFs and the weights of Mignone & Del Zanna (2021)
    ap, am = Sr.clamp(min=0.0), Sl.clamp(max=0.0)
    z = 1.0 / (ap - am)
    eb = (ap * vl[1 + t] - am * vr[1 + t]) * z
    et = -(ap * vl[1 + b] - am * vr[1 + b]) * z
    Al, Ar = SM - Bn.abs() / ql, SM + Bn.abs() / qr
    xl = (vl[1 + d] - SM) * (Sl - SM) / (Al + Sl - 2.0 * SM)
    xr = (vr[1 + d] - SM) * (Sr - SM) / (Ar + Sr - 2.0 * SM)
    nl = (Al + Sl) / (Al.abs() + Sl.abs())
    nr = (Ar + Sr) / (Ar.abs() + Sr.abs())
    nm = (Al + Ar) / (Al.abs() + Ar.abs())
    far = (Ar - Al).abs() > 1e-9 * (Sr - Sl).abs()
    wdl = torch.where(far, 0.5 * xl * (nl - nm) + 0.5 * (Al.abs() - nm * Al),
                      0.5 * xl * nl + 0.5 * Al.abs())
    wdr = torch.where(far, 0.5 * xr * (nr - nm) + 0.5 * (Ar.abs() - nm * Ar),
                      0.5 * xr * nr + 0.5 * Ar.abs())
    wal = torch.where(far, 0.5 * (1.0 + nm), torch.full_like(nm, 0.5))
    war = torch.where(far, 0.5 * (1.0 - nm), torch.full_like(nm, 0.5))
    wal, war = torch.where(hll, ap * z, wal), torch.where(hll, -am * z, war)
    wdl, wdr = torch.where(hll, -am * ap * z, wdl), torch.where(hll, -am * ap * z, wdr)
    return f, cmax, {"eb": eb, "et": et, "a": (wal, war), "d": (wdl, wdr)}


def _hllc_hd(vl, vr, d, g):
    ul, ur = _cons_hd(vl, g), _cons_hd(vr, g)

    def flux(v, u):
        f = u * v[1 + d]
        f[0] = u[1 + d]
        f[1 + d] += v[4]
        f[4] = (u[4] + v[4]) * v[1 + d]
        return f
    fl, fr = flux(vl, ul), flux(vr, ur)
    al, ar = torch.sqrt(g * vl[4] / vl[0]), torch.sqrt(g * vr[4] / vr[0])
    Sl = torch.minimum(vl[1 + d] - al, vr[1 + d] - ar)
    Sr = torch.maximum(vl[1 + d] + al, vr[1 + d] + ar)
    dl, dr = vl[1 + d] - Sl, vr[1 + d] - Sr
    vs = (vr[4] + ur[1 + d] * dr - vl[4] - ul[1 + d] * dl) / (vr[0] * dr - vl[0] * dl)
    side = []
    for v, u, S, f in ((vl, ul, Sl, fl), (vr, ur, Sr, fr)):
        r = u[0] * (S - v[1 + d]) / (S - vs)
        s = r * torch.stack([torch.ones_like(r), v[1], v[2], v[3], u[4] / v[0]
                             + (vs - v[1 + d]) * (vs + v[4] / (v[0] * (S - v[1 + d])))])
        s[1 + d] = r * vs
        side.append(f + S * (s - u))
    f = torch.where(vs >= 0, side[0], side[1])
    f = torch.where(Sr < 0, fr, f)
    f = torch.where(Sl > 0, fl, f)
    return f, torch.maximum(Sl.abs(), Sr.abs()), None


def _prim(u, g, mhd):
    v = u.clone()
    v[1:4] = u[1:4] / u[0]
    k = 0.5 * (u[1] ** 2 + u[2] ** 2 + u[3] ** 2) / u[0]
    if mhd:
        k = k + 0.5 * (u[4] ** 2 + u[5] ** 2 + u[6] ** 2)
    p = (g - 1.0) * (u[-1] - k)
    v[-1] = torch.where(p < 0, torch.full_like(p, 1e-12), p)
    u[-1] = torch.where(p < 0, v[-1] / (g - 1.0) + k, u[-1])
    return v


def _half_edge(ct, b, vel, dcoef, along, avg, limiter):
    """Upwind average and dissipation of one face field at the edges."""
    br, bl = _emf_edges(b, along, limiter, True)      # states right and left of a face
    vr, vl = _emf_edges(vel, along, limiter, False)
    bl, vl = _dn(bl, along), _dn(vl, along)
    half = lambda w: 0.5 * (_dn(w, avg) + w)
    aL, aR = (half(w) for w in ct[dcoef]["a"])
    dL, dR = (half(w) for w in ct[dcoef]["d"])
    return aL * vl * bl + aR * vr * br, dR * br - dL * bl


def _stage(V, Bs, h, dt, g, limiter):
    """(cell increments, face increments, inverse time step) of one stage."""
    ndim, mhd = len(h), len(V) == 8
    R, C, ct = None, None, []
    for d in range(ndim):
        lo, hi = _cell_edges(V, d, limiter)
        vl, vr = _dn(hi, d).clone(), lo.clone()
        if mhd:
            vl[4 + d], vr[4 + d] = Bs[d], Bs[d]
            f, cm, c = _hlld(vl, vr, Bs[d], d, g)
            ct.append(c)
        else:
            f, cm, _ = _hllc_hd(vl, vr, d, g)
        r = -dt / h[d] * (_up(f, d) - f)
        c = 0.5 * (cm + _up(cm, d)) / h[d]
        R, C = (r, c) if R is None else (R + r, C + c)
        del lo, hi, vl, vr, f
    if not mhd:
        return R, [], C

    def edge(first, s1, second, s2):
        a1, p1 = _half_edge(ct, *first, limiter)
        a2, p2 = _half_edge(ct, *second, limiter)
        return a1 + s1 * p1 + a2 + s2 * p2
    Ez = edge((Bs[1], ct[1]["et"], 0, 0, 1), 1, (Bs[0], ct[0]["eb"], 1, 1, 0), -1)
    k = [dt / x for x in h]
    if ndim == 2:
        return R, [-k[1] * (_up(Ez, 1) - Ez), k[0] * (_up(Ez, 0) - Ez)], C
    Ey = edge((Bs[2], ct[2]["eb"], 0, 0, 2), -1, (Bs[0], ct[0]["et"], 2, 2, 0), 1)
    Ex = edge((Bs[2], ct[2]["et"], 1, 1, 2), 1, (Bs[1], ct[1]["eb"], 2, 2, 1), -1)
    return R, [-(k[1] * (_up(Ez, 1) - Ez) - k[2] * (_up(Ey, 2) - Ey)),
               k[0] * (_up(Ez, 0) - Ez) - k[2] * (_up(Ex, 2) - Ex),
               -(k[0] * (_up(Ey, 0) - Ey) - k[1] * (_up(Ex, 1) - Ex))], C


def _advance(V, Bs, n, ndim, physics, limiter, rk, steps, dt, cfl):
    g, h, mhd = GAMMA[physics], [1.0 / m for m in n[:ndim]], physics == "mhd"
    U = (_cons_mhd if mhd else _cons_hd)(V, g)
    weights = [(0.5, 0.5)] if rk == 2 else [(0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)]
    for _ in range(steps):
        U0, B0, inv = U, Bs, None
        for stage in range(rk):
            R, rb, C = _stage(V, Bs, h, dt, g, limiter)
            if stage == 0:
                inv = float(C.max()) / ndim
                U, Bs = U0 + R, [b + r for b, r in zip(B0, rb)]
            else:
                a, c = weights[stage - 1]
                U = a * U0 + c * U + c * R
                Bs = [a * b0 + c * b + c * r for b0, b, r in zip(B0, Bs, rb)]
            for d, b in enumerate(Bs):
                U[4 + d] = 0.5 * (b + _up(b, d))
            V = _prim(U, g, mhd)
        dt = min(cfl / inv, 1.1 * dt)
    return V, U, Bs, dt


def exact(case, seed):
    if case["kind"] == "grid":
        # The relativistic solver has no such value: its secant stops part way, at the
        # iterate that its rounding picked.  Open sides: not restated here.
        if case["physics"] == "rmhd" or case["sides"] != "periodic":
            return None
        n, ndim, physics = _shape(case), case["ndim"], case["physics"]
        V, Bs = _inputs(physics, ndim, n, case["ic"], seed)
        V, U, Bs, dt = _advance(V, Bs, n, ndim, physics, case["limiter"], case["rk"],
                                case["steps"], _first_dt(n, ndim, physics), 0.4)
        return {"V": V, "U": U, "B": Bs, "dt": dt}
    out = {"dt": None}
    members = _members(case)
    for g in _due(case):
        physics, n, _ = members[g]
        V, Bs = _inputs(physics, _ndim(n), n, "turbulence", seed * 1000 + g)
        V, U, Bs, _ = _advance(V, Bs, n, _ndim(n), physics, "mc", 2, case["steps"],
                               _first_dt(n, _ndim(n), physics), 0.4)
        out["grid%02d" % g] = [V, U] + Bs
    return out
