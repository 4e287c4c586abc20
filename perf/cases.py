"""The workloads this framework's speed is judged on, each through the public entry points.

Three ways a program uses the framework:

  solve   a whole run from the data files of a run directory: ``Solver(rundir)``, ``run()``
          to the final time, the hierarchy and the values read back (what the reference's
          amr2 / amr3 program does between its input files and its last frame);
  frames  a context that stays on the device and is read back every few coarse steps
          (``run(max_cycles)``, ``values()``), on one uniform level;
  driver  a driver that keeps its own time loop and calls the level entry points
          (``level_advance`` per level and substep, ``update`` after the subcycles), as the
          Fortran binding does, and reads a frame every few coarse steps;
  serve   a burst of independent solves handed to the serving loop.

The problems, options and sizes are the repository's own: the 2D advection, Euler, acoustics
and annulus configurations and the 3D Euler blast and swirl of the tests, the benchmark and
the serving stream, in FP64 and in the FP32 form, unsplit and Godunov-split. The seed moves
what a user would move: positions, radii, velocities, states.
"""
from __future__ import annotations

import dataclasses
import math
import random
import tempfile

import numpy as np
import torch

from amrclaw_b200 import ClawRunData, Solver, problems, serve

MEQN = {"advection2d": 1, "euler2d": 4, "acoustics2d": 3, "annulus2d": 1, "blast3d": 5, "swirl3d": 1}


PROBLEM = {"advection": "advection2d", "euler": "euler2d", "acoustics": "acoustics2d"}  # of the serving stream


def _case(name, kind, problem, n, levels, precision="fp64", **kw):
    c = {"name": name, "kind": kind, "problem": problem, "n": n, "levels": levels, "ratio": 2, "precision": precision,
         "split": False, "tfinal": 0.0, "steps": 0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest: the periodic advection square on its stated base grid for some coarse
        # steps; launches and the host's part count most
        _case("adv2d_50_solve", "solve", "advection2d", 50, 3, tfinal=0.1),
        # the four-quadrant Riemann problem at its stated size: four levels, many small patches
        _case("euler2d_100_solve", "solve", "euler2d", 100, 4, tfinal=0.15),
        # the acoustic pulse in the FP32 form, four levels
        _case("acou2d_64_f32_solve", "solve", "acoustics2d", 64, 4, "fp32", tfinal=0.2),
        # mapped grid: face velocities and a capacity function in aux, a ragged base grid
        _case("annulus2d_solve", "solve", "annulus2d", 20, 3, tfinal=0.2),
        # one large uniform level (a convergence study's reference run), odd tile remainders
        _case("euler2d_1002_frames", "frames", "euler2d", 1002, 1, steps=50),
        # the Godunov-split scheme on a uniform level, FP32
        _case("acou2d_500_split_f32_frames", "frames", "acoustics2d", 500, 1, "fp32", steps=50, split=True),
        # a uniform 3D level as one grid
        _case("blast3d_90_frames", "frames", "blast3d", 90, 1, steps=20),
        # the 3D radial blast at its stated size with three levels: the headline workload
        _case("blast3d_64_solve", "solve", "blast3d", 64, 3, tfinal=0.2),
        # the same flow in the FP32 form on a smaller base grid
        _case("blast3d_40_f32_solve", "solve", "blast3d", 40, 2, "fp32", tfinal=0.25),
        # the swirl in the FP32 form: four levels, face velocities scaled in time
        _case("swirl3d_32_f32_solve", "solve", "swirl3d", 32, 4, "fp32", tfinal=0.15),
        # a driver's own time loop over the level entry points, three levels in 3D
        _case("blast3d_48_driver", "driver", "blast3d", 48, 3, steps=4),
        # independent 2D solves of mixed problems and precisions arriving together
        _case("serve2d_16", "serve", "mixed2d", 64, 3, "mixed", steps=16),
    ]


def _even(x):
    return max(2, 2 * int(round(x / 2)))


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choice(["solve"] * 5 + ["frames"] * 2 + ["driver"] * 2 + ["serve"])
    if kind == "serve":
        c = _case("", "serve", "mixed2d", _even(_log(rng, 32, 80)), rng.randint(2, 3), "mixed", steps=rng.randint(4, 16))
    elif kind == "frames":
        p = rng.choice(["euler2d", "acoustics2d", "advection2d", "blast3d"])
        n = _even(_log(rng, 64, 1000)) if p != "blast3d" else _even(_log(rng, 16, 80))
        c = _case("", kind, p, n, 1, rng.choice(["fp64", "fp32"]), steps=rng.randint(10, 40) if p != "blast3d" else rng.randint(5, 20),
                  split=p != "blast3d" and rng.random() < 0.3)
    elif kind == "driver":
        p = rng.choice(["blast3d", "acoustics2d", "advection2d"])
        n = _even(_log(rng, 40, 256)) if p != "blast3d" else _even(_log(rng, 16, 48))
        c = _case("", kind, p, n, rng.randint(2, 3), rng.choice(["fp64", "fp32"]), steps=rng.randint(2, 4))
    else:
        p = rng.choice(["advection2d", "euler2d", "acoustics2d", "annulus2d", "blast3d", "blast3d", "swirl3d"])
        prec = "fp64" if p == "annulus2d" else rng.choice(["fp64", "fp32"])
        if p == "blast3d":
            c = _case("", kind, p, _even(_log(rng, 16, 56)), rng.randint(2, 3), prec, tfinal=round(rng.uniform(0.05, 0.2), 3))
        elif p == "swirl3d":
            c = _case("", kind, p, _even(_log(rng, 16, 32)), rng.randint(2, 3), prec, tfinal=round(rng.uniform(0.05, 0.15), 3))
        elif p == "annulus2d":
            c = _case("", kind, p, _even(_log(rng, 16, 40)), rng.randint(2, 3), prec, tfinal=round(rng.uniform(0.1, 0.3), 3))
        else:
            c = _case("", kind, p, _even(_log(rng, 32, 128)), rng.randint(2, 3), prec, tfinal=round(rng.uniform(0.05, 0.2), 3),
                      split=rng.random() < 0.15)
            c["ratio"] = 4 if c["levels"] == 2 and rng.random() < 0.3 else 2
    del c["name"]
    return c


# ------------------------------------------------------------------ run data

def _annulus(n, levels, tfinal, x1):
    rd = ClawRunData(num_dim=2)
    p = rd.probdata
    p.add_param("problem", "advection_annulus")
    for key, val in (("A1", 1.0), ("beta1", 40.0), ("x1", x1), ("y1", 0.0), ("A2", -1.0), ("beta2", 40.0), ("x2", 0.5), ("y2", 0.0)):
        p.add_param(key, val)
    c = rd.clawdata
    c.lower = [0.2, 0.0]; c.upper = [1.0, 2.0 * math.pi]; c.num_cells = [n, 6 * n]
    c.num_eqn = 1; c.num_waves = 1; c.num_aux = 3; c.capa_index = 3
    c.output_style = 1; c.num_output_times = 1; c.tfinal = tfinal; c.output_t0 = False
    c.dt_variable = True; c.dt_initial = 0.1 / n; c.dt_max = 1e99; c.cfl_desired = 0.9; c.cfl_max = 1.0
    c.steps_max = 1000000; c.order = 2; c.transverse_waves = 2; c.limiter = ["vanleer"]
    c.bc_lower = ["extrap", "periodic"]; c.bc_upper = ["extrap", "periodic"]
    a = rd.amrdata
    r = [2] * max(1, levels - 1)
    a.amr_levels_max = levels; a.refinement_ratios_x = list(r); a.refinement_ratios_y = list(r); a.refinement_ratios_t = list(r)
    a.aux_type = ["xleft", "yleft", "capacity"]
    a.flag2refine = True; a.flag2refine_tol = 0.02; a.regrid_interval = 2; a.regrid_buffer_width = 3
    a.clustering_cutoff = 0.7
    return rd


def _blast(n, levels, tfinal, centre, pin):
    rd = ClawRunData(num_dim=3)
    p = rd.probdata
    p.add_param("problem", "euler_blast")
    p.add_param("gamma", 1.4)
    for key, val in zip(("x0", "y0", "z0"), centre):
        p.add_param(key, val)
    p.add_param("r0", 0.2); p.add_param("pin", pin); p.add_param("pout", 1.0); p.add_param("flag_pressure", 1)
    c = rd.clawdata
    c.lower = [-1.0] * 3; c.upper = [1.0] * 3; c.num_cells = [n, n, n]
    c.num_eqn = 5; c.num_waves = 3; c.num_aux = 0
    c.output_style = 1; c.num_output_times = 1; c.tfinal = tfinal; c.output_t0 = False
    c.dt_variable = True; c.dt_initial = 0.2 / n; c.dt_max = 1e99; c.cfl_desired = 0.9; c.cfl_max = 1.0
    c.steps_max = 1000000; c.order = 2; c.transverse_waves = 22; c.limiter = ["mc"] * 3
    c.bc_lower = ["extrap"] * 3; c.bc_upper = ["extrap"] * 3
    a = rd.amrdata
    a.amr_levels_max = levels
    r = [2] * max(1, levels - 1)
    a.refinement_ratios_x = list(r); a.refinement_ratios_y = list(r); a.refinement_ratios_z = list(r); a.refinement_ratios_t = list(r)
    a.flag2refine = True; a.flag2refine_tol = 0.2; a.regrid_interval = 2; a.regrid_buffer_width = 2
    a.clustering_cutoff = 0.7
    a.max1d = 68
    return rd


def _params(case, seed):
    r = random.Random(seed)
    u = r.uniform
    return {"advection2d": lambda: dict(u=u(0.4, 0.6), v=u(0.8, 1.1), x0=(x := u(0.05, 0.3)), x1=x + 0.4, y0=(y := u(0.05, 0.3)), y1=y + 0.4),
            "euler2d": lambda: dict(xs=u(0.7, 0.82), ys=u(0.7, 0.82)),
            "acoustics2d": lambda: dict(r0=u(0.25, 0.35), width=u(0.05, 0.06)),
            "annulus2d": lambda: dict(x1=u(-0.55, -0.45)),
            "blast3d": lambda: dict(centre=[u(-0.1, 0.1) for _ in range(3)], pin=u(4.8, 5.2)),
            "swirl3d": lambda: dict(x0=u(0.45, 0.55), y0=u(0.22, 0.28), z0=u(0.45, 0.55))}[case["problem"]]()


FAR = 1.0e6  # final time of the cases that are read back every few steps


def _rundata(case, seed):
    n, lev, rat, p = case["n"], case["levels"], case["ratio"], case["problem"]
    tf = case["tfinal"] if case["kind"] == "solve" else FAR
    k = _params(case, seed)
    if p == "advection2d":
        rd = problems.advection_square(n, lev, rat, tf, **k)
    elif p == "euler2d":
        rd = problems.euler_quadrants(n, lev, rat, tf, **k)
    elif p == "acoustics2d":
        rd = problems.acoustics_pulse(n, lev, rat, tf, **k)
    elif p == "annulus2d":
        rd = _annulus(n, lev, tf, **k)
    elif p == "blast3d":
        rd = _blast(n, lev, tf, **k)
    else:
        rd = problems.advection_swirl3d(n, lev, rat, tf, vel_period=1.5, **k)
    if case["split"]:
        rd.clawdata.dimensional_split = 1
    if case["kind"] != "solve":
        rd.clawdata.steps_max = 1000000000
    if case["kind"] == "frames":
        rd.amrdata.max1d = n + 4  # the uniform level as one grid
    return rd


def _requests(case, seed):
    """A burst in the manner of the serving stream: the problems in turn, FP64 and FP32 in turn."""
    r = random.Random(case["n"])  # the base grids belong to the case, the flows to the seed
    out = []
    for k in range(case["steps"]):
        kind = serve.KINDS[k % 3]
        key = PROBLEM[kind]
        n = _even(case["n"] * r.uniform(0.75, 1.25))
        out.append(serve.Request(k, 0.0, kind, n, case["levels"], 2, 0.05, "fp32" if (k // 3) % 2 else "fp64",
                                 _params({"problem": key}, seed * 1000 + k)))
    return out


# ------------------------------------------------------------------ the passes

ROWS = 8192  # most grids of a frame


def _room(case, problem, n):
    """Most values of a frame: the base level and a generous share of the domain at each finer one."""
    dim = 3 if problem.endswith("3d") else 2
    base = (6 if problem == "annulus2d" else 1) * n ** dim * MEQN[problem]
    share = [1.0] + ([0.6] * 3 if dim == 2 else [0.5, 0.3, 0.15])
    return int(base * sum(share[lev] * case["ratio"] ** (dim * lev) for lev in range(case["levels"]))) + 4096


class _Frame:
    """The arrays a program keeps for its frames. How many grids and cells there are is a run's own outcome: the
    rest of the arrays is zero."""

    def __init__(self, room, dim):
        self.values, self.grids, self.used = np.zeros(room), np.zeros((ROWS, 2 + 2 * dim), np.int32), [0, 0]

    def take(self, grids, values):
        for array, new, k in ((self.grids, grids, 0), (self.values, values, 1)):
            if len(new) > len(array):
                raise ValueError("a frame of %d rows, room for %d" % (len(new), len(array)))
            array[:len(new)] = new
            array[len(new):max(self.used[k], len(new))] = 0
            self.used[k] = len(new)


WARM = 8  # coarse steps a driver's hierarchy has behind it: the refined levels have settled


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "serve":
        state["requests"] = _requests(case, seed)
        state["frames"] = [_Frame(_room(case, PROBLEM[r.kind], r.n), 2) for r in state["requests"]]
        return state
    dim = 3 if case["problem"].endswith("3d") else 2
    state["frame"] = _Frame(_room(case, case["problem"], case["n"]), dim)
    state["dir"] = tempfile.TemporaryDirectory(prefix="amrcase_")
    _rundata(case, seed).write(state["dir"].name)
    if case["kind"] in ("frames", "driver"):
        state["solver"] = Solver(state["dir"].name, precision=case["precision"])
    if case["kind"] == "driver":
        state["solver"].run(WARM)
        state["lfine"] = int(state["solver"].info()["lfine"])
    return state


def _coarse_step(s, level, lfine):
    """The reference's recursion (tick.f) with a ratio of two in time and no regrid."""
    dt, cfl = s.level_advance(level)
    if level < lfine:
        for _ in range(2):
            _coarse_step(s, level + 1, lfine)
        s.update(level)
    return dt, cfl


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        with Solver(state["dir"].name, precision=case["precision"]) as s:
            s.run()
            f = state["frame"]
            f.take(s.grids(), s.values())
            return {"grids": f.grids, "values": f.values, "mass": s.mass()}
    if case["kind"] == "frames":
        s = state["solver"]
        s.run(case["steps"])
        return {"values": s.values()}
    if case["kind"] == "driver":
        s = state["solver"]
        for _ in range(case["steps"]):
            dt, cfl = _coarse_step(s, 1, state["lfine"])
        f = state["frame"]
        f.take(s.grids(), s.values())
        return {"grids": f.grids, "values": f.values, "dt": dt, "cfl": cfl}
    reqs = [dataclasses.replace(r) for r in state["requests"]]
    out = serve.serve(reqs, budget_bytes=16 << 30, slots=8, keep_values=True)
    for f, r in zip(state["frames"], out["results"]):
        f.take(np.zeros((0, 6), np.int32), r.values)
    return {"values": [f.values for f in state["frames"]], "cells": [float(r.cell_updates) for r in out["results"]],
            "mass": [r.mass for r in out["results"]]}


# ------------------------------------------------------------------ the least work of a pass

# flops of one cell-update of the unsplit method (the split one solves no transverse problems)
FLOPS = {"advection2d": 60.0, "euler2d": 1300.0, "acoustics2d": 300.0, "annulus2d": 80.0, "blast3d": 7000.0, "swirl3d": 300.0}
# largest wave speed: coarse steps are about 0.9 dx / speed long
SPEED = {"advection2d": 1.1, "euler2d": 2.4, "acoustics2d": 2.0, "annulus2d": 2.0, "blast3d": 2.2, "swirl3d": 2.0}
# share of the domain that the refined levels cover, about
COVER = {"advection2d": 0.25, "euler2d": 0.2, "acoustics2d": 0.3, "annulus2d": 0.2, "blast3d": 0.06, "swirl3d": 0.05}


def _updates(case, problem, n, tfinal):
    """(cell-updates of a pass, cells at its end), about: the base level and the share of the refined ones."""
    dim = 3 if problem.endswith("3d") else 2
    base = (6 if problem == "annulus2d" else 1) * float(n) ** dim
    width = 2.0 if problem in ("acoustics2d", "blast3d") else 0.8 if problem == "annulus2d" else 1.0
    steps = case["steps"] if case["kind"] in ("frames", "driver") else max(1.0, tfinal * SPEED[problem] * n / (0.9 * width))
    ups = cells = 0.0
    for lev in range(case["levels"]):
        share = 1.0 if lev == 0 else COVER[problem]
        at = base * share * float(case["ratio"]) ** (dim * lev)
        ups += at * steps * float(case["ratio"]) ** lev
        cells += at
    return ups, cells


def work(case):
    """Every cell-update reads the cell's state once and writes it once; the frame goes out once."""
    if case["kind"] == "serve":
        jobs = [(PROBLEM[serve.KINDS[k % 3]], 4 if (k // 3) % 2 else 8, 0.05) for k in range(case["steps"])]
    else:
        jobs = [(case["problem"], 4 if case["precision"] == "fp32" else 8, case["tfinal"])]
    b = f = 0.0
    for p, size, tf in jobs:
        ups, cells = _updates(case, p, case["n"], tf)
        aux = 2 if p == "annulus2d" else 3 if p == "swirl3d" else 0
        b += ups * (2 * MEQN[p] + aux) * size + cells * MEQN[p] * 8
        f += ups * FLOPS[p] * (0.5 if case["split"] else 1.0)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit values

def _sqsum(q, idx):
    return sum(q[i] * q[i] for i in idx)


class _Euler:
    """Roe solver with the Harten-Hyman fix (one momentum component per space dimension)."""

    def __init__(self, dim):
        self.g1, self.gam, self.dim = 0.4, 1.4, dim

    def roe(self, l, r):
        e, mom = self.dim + 1, range(1, self.dim + 1)
        sl, sr = l[0].sqrt(), r[0].sqrt()
        pl = self.g1 * (l[e] - 0.5 * _sqsum(l, mom) / l[0])
        pr = self.g1 * (r[e] - 0.5 * _sqsum(r, mom) / r[0])
        rs = sl + sr
        u = [None] + [(l[m] / sl + r[m] / sr) / rs for m in mom]
        h = ((l[e] + pl) / sl + (r[e] + pr) / sr) / rs
        u2 = sum(x * x for x in u[1:])
        a2 = self.g1 * (h - 0.5 * u2)
        return u, h, u2, a2.sqrt(), self.g1 / a2

    def waves(self, roe, d, n):
        """Waves and speeds of the jump d in direction n (1-based); the middle ones travel together."""
        u, h, u2, a, g1a2 = roe
        e = self.dim + 1
        a3 = g1a2 * ((h - u2) * d[0] + sum(u[m] * d[m] for m in range(1, e)) - d[e])
        a5 = (d[n] + (a - u[n]) * d[0] - a * a3) / (2 * a)
        a1 = d[0] - a3 - a5
        w1, w2, w3 = [a1], [a3], [a5]
        shear = 0.0
        for m in range(1, e):
            if m == n:
                w1.append(a1 * (u[n] - a)); w2.append(a3 * u[n]); w3.append(a5 * (u[n] + a))
            else:
                t = d[m] - u[m] * d[0]
                w1.append(a1 * u[m]); w2.append(a3 * u[m] + t); w3.append(a5 * u[m])
                shear = shear + t * u[m]
        w1.append(a1 * (h - u[n] * a)); w2.append(a3 * 0.5 * u2 + shear); w3.append(a5 * (h + u[n] * a))
        return [torch.stack(w) for w in (w1, w2, w3)], [u[n] - a, u[n], u[n] + a], shear

    def rpn(self, l, r, n):
        roe = self.roe(l, r)
        d, e = r - l, self.dim + 1
        W, S, _ = self.waves(roe, d, n)
        if self.dim == 2:  # four waves: the entropy and the shear wave are limited apart
            m = 3 - n
            u = roe[0]
            t = d[m] - u[m] * d[0]
            sh = torch.zeros_like(d)
            sh[m] = t; sh[e] = t * u[m]
            W = [W[0], W[1] - sh, sh, W[2]]
            S = [S[0], S[1], S[1], S[2]]
        am = sum(torch.clamp(s, max=0.0) * w for s, w in zip(S, W))
        df = sum(s * w for s, w in zip(S, W))

        def c_of(q):
            p = self.g1 * (q[e] - 0.5 * _sqsum(q, range(1, e)) / q[0])
            return q[n] / q[0], (self.gam * p / q[0]).sqrt()

        ul, cl = c_of(l)
        um, cm = c_of(l + W[0])
        sl, sr = ul - cl, um - cm
        left = (sl < 0) & (S[0] > 0) & (sr > 0)
        am = torch.where(left, sl * (sr - S[0]) / (sr - sl) * W[0], am)
        ur, cr = c_of(r)
        um, cm = c_of(r - W[-1])
        sl, sr = um + cm, ur + cr
        right = ~left & (S[-1] < 0) & (sr > 0) & (sl < 0)
        am = torch.where(right, df - sr * (S[-1] - sl) / (sr - sl) * W[-1], am)
        return W, S, am, df - am, roe

    def rpt(self, roe, d, n):
        W, S, _ = self.waves(roe, d, n)
        return (sum(torch.clamp(s, max=0.0) * w for s, w in zip(S, W)),
                sum(torch.clamp(s, min=0.0) * w for s, w in zip(S, W)))


class _Acoustics:
    def __init__(self):
        self.z = self.c = 2.0  # rho = 1, bulk = 4

    def _split(self, d, n):
        a1, a2 = (-d[0] + self.z * d[n]) / (2 * self.z), (d[0] + self.z * d[n]) / (2 * self.z)
        w1, w2 = torch.zeros_like(d), torch.zeros_like(d)
        w1[0] = -a1 * self.z; w1[n] = a1; w2[0] = a2 * self.z; w2[n] = a2
        return w1, w2

    def rpn(self, l, r, n):
        w1, w2 = self._split(r - l, n)
        c = torch.full_like(w1[0], self.c)
        return [w1, w2], [-c, c], -self.c * w1, self.c * w2, None

    def rpt(self, _, d, n):
        w1, w2 = self._split(d, n)
        return -self.c * w1, self.c * w2


class _Advection:
    def __init__(self, u, v):
        self.u = [None, u, v]

    def rpn(self, l, r, n):
        d, u = r - l, self.u[n]
        return [d], [torch.full_like(d[0], u)], min(u, 0.0) * d, max(u, 0.0) * d, None

    def rpt(self, _, d, n):
        return min(self.u[n], 0.0) * d, max(self.u[n], 0.0) * d


def _along(q, ax, lo, hi):
    """Cells lo..hi-1 of space axis ax (1: x, the last one)."""
    return q.narrow(q.dim() - ax, lo, hi - lo)


def _ghosts(q, per):
    for ax in range(1, q.dim()):
        n = q.shape[q.dim() - ax]
        for g in range(2):
            _along(q, ax, g, g + 1).copy_(_along(q, ax, n - 4 + g if per else 2, n - 3 + g if per else 3))
            _along(q, ax, n - 2 + g, n - 1 + g).copy_(_along(q, ax, 2 + g if per else n - 3, 3 + g if per else n - 2))


def _normal(sol, q, ax, dtdx):
    """One sweep over the array: fluctuations, corrections and Roe data at the faces 1..n-3 of its n cells."""
    n = q.shape[q.dim() - ax]
    W, S, am, ap, roe = sol.rpn(_along(q, ax, 0, n - 1), _along(q, ax, 1, n), ax)
    lim = []
    for w, s in zip(W, S):
        wc, wl, wr = _along(w, ax, 1, n - 2), _along(w, ax, 0, n - 3), _along(w, ax, 2, n - 1)
        sc = _along(s, ax, 1, n - 2)
        nn = (wc * wc).sum(0)
        r = torch.where(sc > 0, (wl * wc).sum(0), (wr * wc).sum(0)) / torch.where(nn == 0, torch.ones_like(nn), nn)
        phi = torch.clamp(torch.minimum(torch.minimum((1 + r) / 2, 2 * r), torch.full_like(r, 2.0)), min=0.0)
        lim.append(torch.where(nn == 0, torch.ones_like(nn), phi) * wc)
    S = [_along(s, ax, 1, n - 2) for s in S]
    cq = sum(s.abs() * (1 - s.abs() * dtdx) * w for s, w in zip(S, lim))
    cut = lambda t: _along(t, ax, 1, n - 2) if torch.is_tensor(t) else t  # noqa: E731
    if roe is not None:
        roe = ([None] + [cut(t) for t in roe[0][1:]],) + tuple(cut(t) for t in roe[1:])
    cfl = max(float(s.abs().max()) for s in S) * dtdx
    return cut(am), cut(ap), 0.5 * cq, roe, cfl


def _rings(q, axes, width):
    for ax in axes:
        q = _along(q, ax, width, q.shape[q.dim() - ax] - width)
    return q


def _step2(sol, q, d, split):
    """One step of the unsplit (transverse corrections of both kinds) or the Godunov-split 2D method; q has its ghosts."""
    cfl = 0.0
    if split:
        for ax in (1, 2):
            n = q.shape[q.dim() - ax]
            src = q if ax == 1 else _along(q, 1, 2, q.shape[2] - 2)
            am, ap, cq, _, c = _normal(sol, src, ax, d[ax])
            m = n - 3
            upd = d[ax] * ((_along(am, ax, 1, m) + _along(cq, ax, 1, m)) - (_along(cq, ax, 0, m - 1) - _along(ap, ax, 0, m - 1)))
            _along(src, ax, 2, n - 2).sub_(upd)
            cfl = max(cfl, c)
        return cfl
    F = {}
    for ax in (1, 2):
        o = 3 - ax
        am, ap, cq, roe, c = _normal(sol, _rings(q, [o], 1), ax, d[ax])
        cfl = max(cfl, c)
        m = am.shape[am.dim() - ax]
        a2, p2 = am + 2 * cq, ap - 2 * cq
        bm1, bp1 = sol.rpt(roe, a2, o)
        bm2, bp2 = sol.rpt(roe, p2, o)
        h = 0.5 * d[ax]
        lo = -h * (_along(bm1, ax, 1, m) + _along(bm2, ax, 0, m - 1))
        up = -h * (_along(bp1, ax, 1, m) + _along(bp2, ax, 0, m - 1))
        k = lo.shape[lo.dim() - o]
        F[o, "t"] = _along(up, o, 0, k - 1) + _along(lo, o, 1, k)
        F[ax, "m"], F[ax, "p"] = _rings(am + cq, [o], 1), _rings(cq - ap, [o], 1)
    inner = _rings(q, [1, 2], 2)
    out = inner.clone()
    for ax in (1, 2):
        m = F[ax, "m"].shape[3 - ax]
        out -= d[ax] * (_along(F[ax, "m"] + F[ax, "t"], ax, 1, m) - _along(F[ax, "p"] + F[ax, "t"], ax, 0, m - 1))
    inner.copy_(out)
    return cfl


def _step3(sol, q, d):
    """One step of the unsplit 3D method with transverse_waves 22; q has its ghosts."""
    cfl, F, T = 0.0, {}, {1: 0.0, 2: 0.0, 3: 0.0}
    for ax in (1, 2, 3):
        y, z = ax % 3 + 1, (ax + 1) % 3 + 1
        am, ap, cq, roe, c = _normal(sol, _rings(q, [y, z], 1), ax, d[ax])
        cfl = max(cfl, c)
        m = am.shape[am.dim() - ax]
        F[ax] = (_rings(am + cq, [y, z], 1), _rings(cq - ap, [y, z], 1))
        tot = {}
        for side, f, sg in ((1, am, -1.0), (2, ap, 1.0)):
            sp = {}
            for o in (y, z):
                sp[o] = sol.rpt(roe, f, o), sol.rpt(roe, cq, o)
            part = {}
            for o, t in ((y, z), (z, y)):  # faces of direction o, moved along t
                (bm, bp), (bmq, bpq) = sp[o]
                (cm, cp), (cmq, cpq) = sp[t]
                P1, P2 = sol.rpt(roe, cp - sg * 3 * cpq, o)
                M1, M2 = sol.rpt(roe, cm - sg * 3 * cmq, o)
                e = d[ax] * d[t] / 6.0
                part[o, 1, 0] = -0.5 * d[ax] * bm + e * (P1 - M1) + sg * d[ax] * bmq
                part[o, 2, 0] = -0.5 * d[ax] * bp + e * (P2 - M2) + sg * d[ax] * bpq
                part[o, 1, 1], part[o, 2, 1] = -e * P1, -e * P2
                part[o, 1, -1], part[o, 2, -1] = e * M1, e * M2
            at = (1, m) if side == 1 else (0, m - 1)
            for key, v in part.items():
                v = _along(v, ax, *at)
                tot[key] = v if key not in tot else tot[key] + v
        for (o, side, off), v in tot.items():
            t = y if o == z else z
            n, k = v.shape[v.dim() - o], v.shape[v.dim() - t]
            v = _along(v, o, 1, n) if side == 1 else _along(v, o, 0, n - 1)  # faces between pencils
            T[o] = T[o] + _along(v, t, 1 - off, k - 1 - off)
    inner = _rings(q, [1, 2, 3], 2)
    out = inner.clone()
    for ax in (1, 2, 3):
        m = F[ax][0].shape[4 - ax]
        out -= d[ax] * (_along(F[ax][0] + T[ax], ax, 1, m) - _along(F[ax][1] + T[ax], ax, 0, m - 1))
    inner.copy_(out)
    return cfl


def _initial(case, k, X):
    if case["problem"] == "advection2d":
        x, y = X
        inside = (x > k["x0"]) & (x < k["x1"]) & (y > k["y0"]) & (y < k["y1"])
        return torch.stack([0.1 + 0.9 * inside.to(torch.float64)])
    if case["problem"] == "acoustics2d":
        r = (X[0] * X[0] + X[1] * X[1]).sqrt()
        p = torch.exp(-((r - k["r0"]) / k["width"]) ** 2)
        return torch.stack([p, torch.zeros_like(p), torch.zeros_like(p)])
    if case["problem"] == "euler2d":
        e, n = X[0] >= k["xs"], X[1] >= k["ys"]

        def pick(ne, nw, sw, se):
            v = [torch.full(n.shape, t, dtype=torch.float64, device=n.device) for t in (ne, nw, sw, se)]
            return torch.where(n, torch.where(e, v[0], v[1]), torch.where(e, v[3], v[2]))

        rho, u = pick(1.5, 0.532258064516129, 0.137992831541219, 0.532258064516129), pick(0.0, 1.206045378311055, 1.206045378311055, 0.0)
        v, p = pick(0.0, 0.0, 1.206045378311055, 1.206045378311055), pick(1.5, 0.3, 0.029032258064516, 0.3)
        return torch.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])
    r = sum((x - c) ** 2 for x, c in zip(X, k["centre"])).sqrt()
    p = 1.0 + (k["pin"] - 1.0) * (r <= 0.2).to(torch.float64)
    z = torch.zeros_like(p)
    return torch.stack([torch.ones_like(p), z, z, z, p / 0.4])


def exact(case, seed):
    """The uniform-level frames in 64 bits. An adaptive hierarchy's values have none: what is refined, and so
    where values live, is the run's own outcome."""
    if case["kind"] != "frames":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p, n, dim = case["problem"], case["n"], 3 if case["problem"] == "blast3d" else 2
    k = _params(case, seed)
    lo, hi = (-1.0, 1.0) if p in ("acoustics2d", "blast3d") else (0.0, 1.0)
    dx = (hi - lo) / n
    x = lo + (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) * dx
    X = [x.view([-1 if i == dim - 1 - a else 1 for i in range(dim)]).expand([n] * dim) for a in range(dim)]
    sol = _Euler(dim) if p in ("euler2d", "blast3d") else _Acoustics() if p == "acoustics2d" else _Advection(k["u"], k["v"])
    q0 = _initial(case, k, X)
    q = torch.zeros([MEQN[p]] + [n + 4] * dim, dtype=torch.float64, device=dev)
    _rings(q, range(1, dim + 1), 2).copy_(q0)
    dt = {"advection2d": 0.4, "euler2d": 0.05, "acoustics2d": 0.5, "blast3d": 0.2}[p] / n
    for _ in range(case["steps"]):
        _ghosts(q, p == "advection2d")
        d = [None] + [dt / dx] * dim
        c = _step3(sol, q, d) if dim == 3 else _step2(sol, q, d, case["split"])
        dt = dt * 0.9 / c
    return {"values": _rings(q, range(1, dim + 1), 2).reshape(-1).cpu()}
