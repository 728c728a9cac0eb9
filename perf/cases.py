"""The calls a user of csu_b200 waits for, at the sizes they are made at: whole solver calls through the Python
view of the C ABI (Engine, Pack), from the state in host memory to the state back in host memory.

Four kinds of call:
    solve     one steady solve advanced by `iters` iterations (RK, LU-SGS or DPLUR)
    tube      the unsteady shock tube run to its end time
    pack      several solves advanced together, as the serving loop does
    residual  one residual evaluation, for a caller with a time integrator of its own

Meshes are those of csu_b200.meshgen. The initial states are the free stream (or the Sod states) with smooth
seeded disturbances of every variable, so that gradients, limiters and upwind switches all have work to do.
"""
import functools
import math

import numpy as np
import torch

from csu_b200 import Case, Engine, Pack, Prep, meshgen

NVAR = {"euler": 4, "laminar": 4, "sa": 5, "sst": 6}


def _solve(name, geo, cells, model, **kw):
    c = {"name": name, "kind": "solve", "geo": geo, "cells": cells, "model": model, "scheme": "DPLUR",
         "flux": "AUSM", "order": 2, "stages": 5, "sweeps": 4, "fp32": False, "local": False, "cfl": 5.0,
         "limiter": 0, "limk": 5.0, "iters": 20}
    c.update(kw)
    return c


def listed():
    return [
        # the Sod tube: the smallest unsteady run, about a thousand steps of a few thousand cells (launch latency)
        {"name": "sod_tube", "kind": "tube", "ni": 1000},
        # the reference's own example cases: 2,800 to 12,000 cells, RK5, AUSMDV, second order, CFL 1
        _solve("channel_rk5", "bump", 3139, "euler", scheme="RK", flux="AUSMDV", cfl=1.0, limk=1.0, iters=50),
        # its implicit example: LU-SGS on a 6,000-cell wedge
        _solve("wedge_lusgs", "ramp", 5966, "euler", scheme="LUSGS", flux="AUSMDV", cfl=10.0, limk=1.0, iters=50),
        # laminar boundary-layer case of ordinary size, mixed triangles and quads, RK5
        _solve("bump_laminar_rk5", "bump", 30011, "laminar", scheme="RK", flux="AUSMDV", cfl=1.0, limk=1.0, iters=20),
        # the compression ramp the benchmark runs: 160,000 triangles, FP64 DPLUR with 4 sweeps
        _solve("ramp_dplur", "ramp", 160000, "euler"),
        # the same mesh a step at a time, as a coupled program with the state on the host calls it
        _solve("ramp_step", "ramp", 160000, "euler", iters=1),
        # a fine mesh: nothing fits in L2
        _solve("ramp_dplur_large", "ramp", 500001, "euler", iters=10),
        # the turbulent flat plate, 545 x 385 quads: SA, Roe, Barth-Jespersen, FP32 blocks, 16 sweeps, local steps
        _solve("plate_sa", "plate", 209825, "sa", flux="ROE", limiter=1, fp32=True, local=True, sweeps=16, cfl=1.0,
               iters=8),
        # one request of the serving stream alone: laminar, first order, 16 sweeps, FP32 blocks
        _solve("request_laminar", "bump", 41000, "laminar", order=1, fp32=True, local=True, sweeps=16, cfl=16.0,
               iters=40),
        # six SA requests of the serving stream in one pack
        {"name": "pack_sa", "kind": "pack", "geo": "cylinder", "cells": 24000, "solves": 6, "model": "sa",
         "fp32": True, "sweeps": 16, "cfl": 4.0, "iters": 40},
        # transonic SST airfoils in one pack
        {"name": "pack_sst", "kind": "pack", "geo": "airfoil", "cells": 16384, "solves": 8, "model": "sst",
         "fp32": True, "sweeps": 16, "cfl": 2.0, "iters": 30},
        # one residual for a caller's own time integration
        {"name": "residual", "kind": "residual", "geo": "ramp", "cells": 160000, "flux": "AUSM", "order": 2,
         "limk": 5.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "rk", "rk", "lusgs", "dplur", "dplur", "dplur", "request", "request", "sa", "pack",
                       "residual"])
    if kind == "tube":
        return {"kind": "tube", "ni": _log(rng, 200, 999)}
    if kind == "residual":
        return {"kind": "residual", "geo": rng.choice(["ramp", "bump"]), "cells": _log(rng, 1500, 400000),
                "flux": rng.choice(["ROE", "AUSM"]), "order": rng.choice([1, 2]), "limk": 5.0}
    if kind == "pack":
        model = rng.choice(["laminar", "sa", "sst"])
        solves = rng.randint(2, 8)
        return {"kind": "pack", "geo": "airfoil" if model == "sst" else rng.choice(["bump", "cylinder"]),
                "cells": _log(rng, 5000, 140000 // solves), "solves": solves, "model": model,
                "fp32": rng.random() < 0.75, "sweeps": rng.choice([4, 16]), "cfl": 2.0, "iters": 20}
    if kind == "rk":
        cells = _log(rng, 2500, 60000)
        c = _solve("", "bump", cells, rng.choice(["euler", "laminar", "sa"]), scheme="RK", cfl=1.0, limk=1.0,
                   flux=rng.choice(["AUSM", "AUSMDV"]), stages=rng.choice([3, 4, 5]), iters=20)
    elif kind == "lusgs":
        c = _solve("", rng.choice(["ramp", "bump"]), _log(rng, 3000, 100000), "euler", scheme="LUSGS",
                   flux="AUSMDV", cfl=5.0, limk=1.0, iters=20)
    elif kind == "dplur":
        cells = _log(rng, 1600, 400000)
        c = _solve("", "ramp", cells, "euler", fp32=rng.random() < 0.4, sweeps=rng.choice([4, 4, 5, 20]), cfl=2.0,
                   flux=rng.choice(["ROE", "AUSM", "AUSMDV"]), iters=max(1, min(40, 1500000 // cells)))
    elif kind == "request":
        c = _solve("", rng.choice(["bump", "cylinder"]), _log(rng, 10000, 200000), rng.choice(["laminar", "sa"]),
                   order=1, fp32=rng.random() < 0.6, local=True, sweeps=16, cfl=4.0, iters=10)
    else:
        c = _solve("", "plate", _log(rng, 20000, 150000), "sa", flux=rng.choice(["ROE", "AUSMDV"]), limiter=1,
                   fp32=rng.random() < 0.6, local=True, sweeps=rng.choice([4, 16]), cfl=1.0, iters=6)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=24)
def _case(geo, cells, model, mach, solver, extra):
    """A case read from its SU2 text; the mesh and settings are a program's own and do not change with the seed."""
    visc = None if model == "euler" else model
    kw = dict(solver)
    limk = kw.pop("limk", None)
    re = {"laminar": 1e4, "sa": 2e6, "sst": 6e6}.get(model)
    if geo == "ramp":
        nj = max(4, int(round(math.sqrt(cells / 4.0))))
        ni = max(8, int(round(cells / (2.0 * nj))))
        su2, inp = meshgen.ramp(ni=ni, nj=nj, mach=mach, lim_k=limk or 5.0, **kw)
    else:
        if geo == "bump":
            su2, inp = meshgen.bump(ncells=cells, mach=mach, viscous=visc, re=re, **kw)
        elif geo == "cylinder":
            su2, inp = meshgen.cylinder(ncells=cells, mach=mach, viscous=visc, re=re, **kw)
        elif geo == "airfoil":
            su2, inp = meshgen.airfoil(ncells=cells, mach=mach, alpha_deg=2.0, viscous=visc, re=re, **kw)
        else:
            nj = int(round(math.sqrt(cells * 385 / 545.0)))
            su2, inp = meshgen.plate(ni=int(round(cells / nj)), nj=nj, viscous=visc, **kw)
        if limk:
            inp += "limK, %g\n" % limk
    return Case.from_text(inp + extra, su2)


@functools.lru_cache(maxsize=8)
def _tube(ni):
    su2, inp = meshgen.sod_tube(ni=ni, stages=2)
    return Case.from_text(inp + "limiterFunc, 1\n", su2)


def _case_of(case):
    if case["kind"] == "tube":
        return _tube(case["ni"])
    mach = {"ramp": 2.5, "plate": 0.2, "airfoil": 0.7, "cylinder": 0.6, "bump": 0.5}[case["geo"]]
    if case["kind"] == "residual":
        solver = (("flux", case["flux"]), ("order", case["order"]), ("limk", case["limk"]))
        return _case(case["geo"], case["cells"], "euler", mach, solver, "")
    if case["kind"] == "pack":
        solver = (("flux", "AUSM"), ("order", 1), ("n_linear", case["sweeps"]), ("cfl", case["cfl"]))
        return _case(case["geo"], case["cells"], case["model"], mach, solver,
                     "implicitLocalDt, 1\nimplicitFP32, %d\n" % case["fp32"])
    solver = (("flux", case["flux"]), ("order", case["order"]), ("n_linear", case["sweeps"]), ("cfl", case["cfl"]),
              ("limk", case["limk"]), ("scheme", case["scheme"]))
    extra = "limiterFunc, %d\nimplicitFP32, %d\nimplicitLocalDt, %d\n" % (case["limiter"], case["fp32"], case["local"])
    if case["geo"] == "plate":
        extra += "CFLramp, 300\nCFLmax, 16\n"
    return _case(case["geo"], case["cells"], case["model"], mach, solver, extra)


def _centres(case):
    nodes, n = case.cell_nodes, case.cell_npts
    p = case.xy[np.maximum(nodes, 0)]
    p[nodes < 0] = 0.0
    return p.sum(axis=1) / n[:, None]


def _disturbed(case, seed, amplitude=0.02):
    """The case's initial state with four smooth seeded modes on each of rho, u, v, p and the scalars."""
    rng = np.random.default_rng(seed)
    U = case.initial_state()
    xy = _centres(case)
    lo, hi = xy.min(axis=0), xy.max(axis=0)
    x, y = ((xy - lo) / np.maximum(hi - lo, 1e-300)).T

    def f():
        s = np.zeros(len(x))
        for _ in range(4):
            k = rng.uniform(0.5, 5.0, 2) * rng.choice([-1.0, 1.0], 2)
            s += rng.uniform(0.3, 1.0) * np.sin(2 * math.pi * (k[0] * x + k[1] * y + rng.uniform()))
        return amplitude * s / 2.5

    g = case.config.gamma - 1.0
    r, u, v = U[0], U[1] / U[0], U[2] / U[0]
    k = U[4] / r if len(U) == 6 else 0.0
    p = g * (U[3] - 0.5 * r * (u * u + v * v) - r * k)
    ref = np.sqrt(u * u + v * v) + 0.1 * np.sqrt(1.4 * p / r)
    X = U[4:] / r
    r, u, v, p = r * (1 + f()), u + ref * f(), v + ref * f(), p * (1 + f())
    X = [X[i] * (1 + f()) for i in range(len(X))]
    k = X[0] if len(U) == 6 else 0.0
    return np.stack([r, r * u, r * v, p / g + 0.5 * r * (u * u + v * v) + r * k] + [r * q for q in X])


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    n = t.numpy()
    n[...] = a
    return t, n


def prepare(case, seed):
    c = _case_of(case)
    if case["kind"] == "pack":
        preps = [Prep(c, state=_disturbed(c, 1000 * seed + i, 0.01)) for i in range(case["solves"])]
        return {"case": case, "preps": preps, "pack": Pack(preps)}
    config = c.config
    if case["kind"] == "tube":
        U = _disturbed(c, seed, 0.005)
    else:
        U = _disturbed(c, seed)
        if case["kind"] == "solve" and case["stages"] != config.stages:
            # the generators write stages 5
            config = type(config).from_buffer_copy(config)
            config.stages = case["stages"]
    hold, host = _pinned(U)
    back, out = _pinned(U)
    return {"case": case, "engine": Engine(c, config=config, state=host), "U0": host, "out": out,
            "tmax": c.get_double("tmax") if case["kind"] == "tube" else 0.0, "hold": (hold, back)}


def run(state):
    case = state["case"]
    if case["kind"] == "pack":
        pack = state["pack"]
        for k, p in enumerate(state["preps"]):
            pack.set_state(k, p.state)
        pack.iterate(case["iters"])
        info = [pack.info(k) for k in range(len(pack))]
        return {"U": [pack.get_state(k) for k in range(len(pack))], "res": [i["res"] for i in info],
                "coef": [i["coef"] for i in info], "status": [i["status"] for i in info]}
    eng = state["engine"]
    eng.set_state(state["U0"])
    if case["kind"] == "residual":
        return {"R": eng.residual()}
    if case["kind"] == "tube":
        steps, t = eng.tube_run(state["tmax"])
        return {"steps": steps, "t": t, "U": eng.get_state(out=state["out"])}
    hist = eng.iterate(case["iters"])
    return {"hist": hist, "U": eng.get_state(out=state["out"])}


def work(case):
    """Per residual evaluation and update of a cell: the state read and written once, the mesh (node coordinates,
    connectivity, volumes) read once; the DPLUR operator's blocks are intermediate values and are not counted.
    Operations: least-squares gradients, limiters, fluxes and updates; per sweep the block products."""
    nv = NVAR[case.get("model", "euler")]
    cells = case["cells"] * case.get("solves", 1) if "cells" in case else 4 * case["ni"]
    faces = 2.0 if case.get("geo") in ("cylinder", "airfoil", "plate") else 1.6
    per_cell = 2 * 8 * nv + faces * (16 + 8) + 16 + 8
    if case["kind"] == "residual":
        evals = 1
    elif case["kind"] == "tube":
        evals = 2 * case["ni"]
    else:
        evals = case["iters"] * (case["stages"] if case.get("scheme") == "RK" else 1)
    flops = 60.0 * nv + faces * (60.0 + 10.0 * nv) + (60.0 * nv if case.get("order", 1) == 2 else 0.0)
    if case["kind"] in ("solve", "pack") and case.get("scheme", "DPLUR") != "RK":
        sweeps = case["sweeps"] if case.get("scheme", "DPLUR") == "DPLUR" else 2
        flops += sweeps * 2.0 * faces * 2.0 * nv * nv + 2.0 * faces * 12.0 * nv * nv
    return {"bytes": float(cells * evals * per_cell), "flops": float(cells * evals * flops)}


# ------------------------------------------------------------------------------------------------ exact values

class _Euler:
    """The second-order finite-volume residual of the Euler equations in numpy: least-squares gradients,
    limiter, MUSCL states, Roe, AUSM or AUSMDV fluxes, first-order boundary fluxes."""

    def __init__(self, c, flux, order, limiter, limk):
        self.c, self.flux, self.order, self.limiter, self.limk = c, flux, order, limiter, limk
        cfg, xy = c.config, c.xy
        self.g, self.Rg = cfg.gamma, cfg.gas_r
        self.pin, self.pout, self.efix = np.array(cfg.pin[:4]), cfg.p_out, cfg.e_fix
        nodes, n = c.cell_nodes, c.cell_npts
        self.xc = _centres(c)
        quad = n == 4
        P = xy[np.maximum(nodes, 0)]

        def tri(a, b, d):
            return 0.5 * ((b[:, 0] - a[:, 0]) * (d[:, 1] - a[:, 1]) - (d[:, 0] - a[:, 0]) * (b[:, 1] - a[:, 1]))
        self.vol = tri(P[:, 0], P[:, 1], P[:, 2]) + np.where(quad, tri(P[:, 2], P[:, 3], P[:, 0]), 0.0)
        self.e = c.con[:, :2]
        a, b = xy[c.con[:, 2]], xy[c.con[:, 3]]
        self.S, self.mid = np.stack([b[:, 1] - a[:, 1], a[:, 0] - b[:, 0]], 1), 0.5 * (a + b)
        self.own = c.bface[:, 2]
        a, b = xy[c.bface[:, 0]], xy[c.bface[:, 1]]
        self.Sb, self.midb = np.stack([b[:, 1] - a[:, 1], a[:, 0] - b[:, 0]], 1), 0.5 * (a + b)
        self.flag = np.repeat(c.marker_flag, c.marker_nbf)
        self.nc = c.n_cells
        cell = np.concatenate([self.e[:, 0], self.e[:, 1], self.own])
        S = np.abs(np.concatenate([self.S, self.S, self.Sb]))
        self.sh = np.stack([np.bincount(cell, S[:, k], self.nc) for k in (0, 1)], 1) * 0.5
        # (cell, neighbour) pairs sorted by cell: offsets to the neighbour and to the face, normal equations
        e0, e1, own, xc = self.e[:, 0], self.e[:, 1], self.own, self.xc
        self.by = np.argsort(cell, kind="stable")
        self.cell = cell[self.by]
        self.start = np.searchsorted(self.cell, np.arange(self.nc))
        self.at = np.empty(len(cell), np.int64)
        self.at[self.by] = np.arange(len(cell))
        self.d = np.concatenate([xc[e1] - xc[e0], xc[e0] - xc[e1], self.midb - xc[own]])[self.by]
        self.r = np.concatenate([self.mid - xc[e0], self.mid - xc[e1], self.midb - xc[own]])[self.by]
        self.aa, self.bb, self.cc = (np.add.reduceat(w, self.start) for w in (
            self.d[:, 0] ** 2, self.d[:, 0] * self.d[:, 1], self.d[:, 1] ** 2))
        self.det = self.aa * self.cc - self.bb * self.bb

    def prim(self, U):
        r, u, v = U[0], U[1] / U[0], U[2] / U[0]
        return np.stack([r, u, v, (self.g - 1) * (U[3] - 0.5 * r * (u * u + v * v))])

    def steps(self, U):
        P = self.prim(U)
        a = np.sqrt(self.g * P[3] / P[0])
        return self.vol / ((np.abs(P[1]) + a) * self.sh[:, 0] + (np.abs(P[2]) + a) * self.sh[:, 1])

    def outside(self, P, n):
        """Ghost primitives of the boundary faces, as the reference's boundaryCalcPrimitive gives them."""
        r, u, v, p = P
        a = np.sqrt(self.g * p / r)
        vn = n[0] * u + n[1] * v
        sub = np.sqrt(u * u + v * v) / a < 1
        G = np.stack([r, u - vn * n[0], v - vn * n[1], p])
        ra, ua, va, pa = self.pin
        pb = 0.5 * (pa + p - r * a * (n[0] * (ua - u) + n[1] * (va - v)))
        inlet = np.stack([ra + (pb - pa) / (a * a), ua - n[0] * (pa - pb) / (r * a),
                          va - n[1] * (pa - pb) / (r * a), pb])
        inlet = np.where(sub, inlet, self.pin[:, None])
        po = self.pout
        outlet = np.stack([r + (po - p) / (a * a), u + n[0] * (p - po) / (r * a),
                           v + n[1] * (p - po) / (r * a), po + 0 * p])
        outlet = np.where(sub, outlet, P)
        pw = p + r * a * vn
        wall = np.stack([r + (pw - p) / (a * a), u - n[0] * vn, v - n[1] * vn, pw])
        f = self.flag
        return np.where(f == 0, G, np.where(f == 1, inlet, np.where(f == 2, outlet, wall)))

    def riemann(self, L, R):
        g = self.g
        rL, uL, vL, pL = L
        rR, uR, vR, pR = R
        EL, ER = pL / (g - 1) + 0.5 * rL * (uL * uL + vL * vL), pR / (g - 1) + 0.5 * rR * (uR * uR + vR * vR)
        HL, HR = (EL + pL) / rL, (ER + pR) / rR
        if self.flux == "AUSM":
            cL, cR = np.sqrt(g * pL / rL), np.sqrt(g * pR / rR)
            ML, MR = uL / cL, uR / cR
            with np.errstate(divide="ignore", invalid="ignore"):
                Mp = np.where(np.abs(ML) >= 1, 0.5 * (ML + np.abs(ML)), 0.25 * (ML + 1) ** 2)
                Pp = np.where(np.abs(ML) >= 1, Mp / ML, 0.25 * (ML + 1) ** 2 * (2 - ML))
                Mm = np.where(np.abs(MR) >= 1, 0.5 * (MR - np.abs(MR)), -0.25 * (MR - 1) ** 2)
                Pm = np.where(np.abs(MR) >= 1, Mm / MR, 0.25 * (MR - 1) ** 2 * (2 + MR))
            M, p = Mp + Mm, Pp * pL + Pm * pR
            m = np.where(M > 0, rL * cL, rR * cR) * M
            up = M > 0
            return np.stack([m, m * np.where(up, uL, uR) + p, m * np.where(up, vL, vR), m * np.where(up, HL, HR)])
        if self.flux == "AUSMDV":
            cL, cR = np.sqrt(g * pL / rL), np.sqrt(g * pR / rR)
            cm = np.maximum(cL, cR)
            al, ar = 2 * (pL / rL) / (pL / rL + pR / rR), 2 * (pR / rR) / (pL / rL + pR / rR)
            with np.errstate(divide="ignore", invalid="ignore"):
                h = 0.5 * (uL + np.abs(uL))
                up = np.where(np.abs(uL) < cm, al * (0.25 * (uL + cm) ** 2 / cm - h) + h, h)
                pp = pL * np.where(np.abs(uL) < cm, 0.25 * (uL + cm) ** 2 * (2 - uL / cm) / cm ** 2, h / uL)
                h = 0.5 * (uR - np.abs(uR))
                um = np.where(np.abs(uR) < cm, ar * (-0.25 * (uR - cm) ** 2 / cm - h) + h, h)
                pm = pR * np.where(np.abs(uR) < cm, 0.25 * (uR - cm) ** 2 * (2 + uR / cm) / cm ** 2, h / uR)
            ru = up * rL + um * rR

            def upwind(a, b):
                return 0.5 * (ru * (b + a) - np.abs(ru) * (b - a))
            s = 0.5 * np.minimum(1, 10 * np.abs(pR - pL) / np.minimum(pL, pR))
            f = np.stack([ru, pp + pm + (0.5 + s) * (up * rL * uL + um * rR * uR) + (0.5 - s) * upwind(uL, uR),
                          upwind(vL, vR), upwind(HL, HR)])
            A, B = (uL - cL < 0) & (uR - cR > 0), (uL + cL < 0) & (uR + cR > 0)
            w = 0.125 * np.where(A & ~B, (uR - cR) - (uL - cL), np.where(B & ~A, (uR + cR) - (uL + cL), 0.0))
            one = np.ones_like(uL)
            return f - w * (rR * np.stack([one, uR, vR, HR]) - rL * np.stack([one, uL, vL, HL]))
        sL, sR = np.sqrt(rL), np.sqrt(rR)
        u, v, H = [(sL * x + sR * y) / (sL + sR) for x, y in ((uL, uR), (vL, vR), (HL, HR))]
        a = np.sqrt((g - 1) * (H - 0.5 * (u * u + v * v)))
        d1, d2, d3, d5 = rR - rL, rR * uR - rL * uL, rR * vR - rL * vL, ER - EL
        a4 = ((H - (u * u + v * v)) * d1 + u * d2 + v * d3 - d5) * (g - 1) / (a * a)
        a2 = d3 - d1 * v
        a5, a1 = 0.5 * ((d1 - a4) + (d2 - u * d1) / a), 0.5 * ((d1 - a4) - (d2 - u * d1) / a)

        def fix(x):
            return np.abs(np.where(np.abs(x) < self.efix, 0.5 * (x * x / self.efix + self.efix), x))
        l1, l2, l5 = fix(u - a), fix(u), fix(u + a)
        fL = np.stack([rL * uL, rL * uL * uL + pL, rL * uL * vL, uL * (EL + pL)])
        fR = np.stack([rR * uR, rR * uR * uR + pR, rR * uR * vR, uR * (ER + pR)])
        one, zero = np.ones_like(u), np.zeros_like(u)
        return 0.5 * (fL + fR - a1 * l1 * np.stack([one, u - a, v, H - u * a])
                      - a2 * l2 * np.stack([zero, zero, one, v])
                      - a4 * l2 * np.stack([one, u, v, 0.5 * (u * u + v * v)])
                      - a5 * l5 * np.stack([one, u + a, v, H + u * a]))

    def face(self, L, R, S):
        s = np.hypot(S[:, 0], S[:, 1])
        n = (S / s[:, None]).T

        def turn(Q, sg):
            return np.stack([Q[0], Q[1] * n[0] + sg * Q[2] * n[1], -sg * Q[1] * n[1] + Q[2] * n[0], Q[3]])
        return turn(self.riemann(turn(L, 1), turn(R, 1)), -1) * s

    def residual(self, U):
        """R and the wall pressure-force terms' ghost pressures."""
        P, e, own, nc = self.prim(U), self.e, self.own, self.nc
        sb = np.hypot(self.Sb[:, 0], self.Sb[:, 1])
        nb = (self.Sb / sb[:, None]).T
        Pb = P[:, own]
        G = self.outside(Pb, nb)
        L, R = P[:, e[:, 0]], P[:, e[:, 1]]
        if self.order == 2:
            other = np.concatenate([P[:, e[:, 1]], P[:, e[:, 0]], G], axis=1)[:, self.by]
            cell, start, d, r, nf = self.cell, self.start, self.d, self.r, len(e)
            p0 = self.pin
            q2 = np.array([p0[0] ** 2, p0[1] ** 2 + p0[2] ** 2, p0[1] ** 2 + p0[2] ** 2, p0[3] ** 2])
            eps = (self.limk * np.sqrt(self.vol / self.vol.max())) ** 3
            du = other - P[:, cell]
            A, B = np.add.reduceat(d[:, 0] * du, start, axis=1), np.add.reduceat(d[:, 1] * du, start, axis=1)
            gx, gy = (self.cc * A - self.bb * B) / self.det, (self.aa * B - self.bb * A) / self.det
            hi = np.maximum(P, np.maximum.reduceat(other, start, axis=1)) - P
            lo = np.minimum(P, np.minimum.reduceat(other, start, axis=1)) - P
            d2 = gx[:, cell] * r[:, 0] + gy[:, cell] * r[:, 1]
            d1 = np.where(d2 > 0, hi[:, cell], lo[:, cell])
            with np.errstate(divide="ignore", invalid="ignore"):
                if self.limiter == 1:
                    ph = np.minimum(1.0, d1 / d2)
                else:
                    ee = q2[:, None] * eps[cell]
                    ph = (d1 * d1 + ee + 2 * d2 * d1) / (d1 * d1 + 2 * d2 * d2 + d1 * d2 + ee)
            phi = np.minimum.reduceat(np.where(d2 == 0, 1.0, ph), start, axis=1)
            step = (phi[:, cell] * d2)[:, self.at]
            L, R = L + step[:, :nf], R + step[:, nf:2 * nf]
        F = self.face(L, R, self.S)
        # boundary fluxes: mirror states at symmetry planes, the wall state's own flux at slip walls
        vn = Pb[1] * nb[0] + Pb[2] * nb[1]
        mirror = np.stack([Pb[0], Pb[1] - 2 * vn * nb[0], Pb[2] - 2 * vn * nb[1], Pb[3]])
        Fb = self.face(Pb, np.where(self.flag == 0, mirror, G), self.Sb)
        un = G[1] * nb[0] + G[2] * nb[1]
        H = self.g / (self.g - 1) * G[3] / G[0] + 0.5 * (G[1] ** 2 + G[2] ** 2)
        m = G[0] * un
        free = np.stack([m, m * G[1] + G[3] * nb[0], m * G[2] + G[3] * nb[1], m * H]) * sb
        Fb = np.where(self.flag >= 3, free, Fb)
        out = np.stack([np.bincount(e[:, 0], F[k], nc) - np.bincount(e[:, 1], F[k], nc) + np.bincount(own, Fb[k], nc)
                        for k in range(4)])
        return out, G[3]


RK = {2: (0.5, 1.0), 3: (0.1481, 0.4, 1.0), 4: (0.0833, 0.2069, 0.4265, 1.0), 5: (0.0533, 0.1263, 0.2375, 0.4414, 1.0)}


def exact(case, seed):
    """Residuals, explicit Runge-Kutta runs and tubes of the Euler equations. The implicit operators have no value
    of their own apart from the code's: DPLUR's finite-difference blocks (a step of 1e-6 in the conserved state)
    carry the rounding of the state into the increments, and LU-SGS depends on its colouring."""
    euler = case.get("model", "euler") == "euler"
    if not euler or case["kind"] == "pack" or (case["kind"] == "solve" and case["scheme"] != "RK"):
        return None
    c = _case_of(case)
    if case["kind"] == "residual":
        return {"R": _Euler(c, case["flux"], case["order"], 0, case["limk"]).residual(_disturbed(c, seed))[0]}
    if case["kind"] == "tube":
        if case["ni"] > 700:
            return None  # half a minute
        m, U, stages, cfl = _Euler(c, "ROE", 2, 1, 1.0), _disturbed(c, seed, 0.005), 2, c.config.cfl
        t, tmax = 0.0, c.get_double("tmax")
        while t < tmax:
            dt = cfl * m.steps(U).min()
            last = t + dt > tmax
            dt = tmax - t if last else dt
            V = U
            for a in RK[stages]:
                V = U - dt * 0.5 * stages * a * m.residual(V)[0] / m.vol
            U, t = V, t + dt * stages / 2.0
            if last:
                break
        return {"steps": None, "t": t, "U": U}
    if case["cells"] * case["iters"] > 1500000:
        return None
    m, U = _Euler(c, case["flux"], case["order"], case["limiter"], case["limk"]), _disturbed(c, seed)
    cfg, rows = c.config, []
    wall = m.flag >= 3
    q = 0.5 * cfg.pin[0] * (cfg.pin[1] ** 2 + cfg.pin[2] ** 2)
    for _ in range(case["iters"]):
        dt, V = cfg.cfl * m.steps(U).min(), U
        for a in RK[case["stages"]]:
            R, pg = m.residual(V)
            V = U - dt * 0.5 * case["stages"] * a * R / m.vol
        U = V
        cp = ((pg - cfg.pin[3]) / q)[wall, None] * m.Sb[wall] / cfg.sref
        rows.append(list(np.sqrt((R * R).mean(axis=1))) + [cp[:, 0].sum(), 0.0, cp[:, 1].sum(), 0.0])
    return {"hist": np.array(rows), "U": U}
