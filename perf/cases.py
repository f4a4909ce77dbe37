"""The calls whose time matters to a user of this library, with their inputs.

Every case goes through a public entry point: `solver.Batch` / `solver.Solver` for time
steps, the `cfd_gauss_solve` / `cfd_sip_solve` seams for a host program that replaces only
its inner solves. `listed()` names the standing cases, `draw()` makes more of the same
kinds and ranges, `prepare()` builds what a program holds before the call (a run already
past its impulsive start, its buffers), `run()` is one call, `work()` its compulsory
traffic and arithmetic, `exact()` the value the result approximates where there is one.

Physics (Re, Ri, Pr, grid skew) come from the seed with the distributions of
`workloads.sweep_draws`; sizes and counts come from the case.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from cfd_solver_b200 import _lib
from cfd_solver_b200.grid import cavity, ogrid
from cfd_solver_b200.solver import Batch, Solver, case_params
from cfd_solver_b200.workloads import CONFIGS, cavity_dt, sweep_draws

SEAM_TOL = 0.75e-2  # the reference's inner tolerance


def listed():
    return [
        # the reference program on its default 65 x 65 grid: one call per step, the step's
        # statistics read every step, the fields at the end (what the INP.DAT driver does)
        dict(name="timeloop_og65", kind="timeloop", form="ogrid", n0=65, n1=65, precision="fp64", steps=10),
        # the smallest configuration (65 x 65 cavity), stepped without per-step host work
        dict(name="steps_cav65", kind="steps", form="cavity", n0=65, n1=65, precision="fp64", steps=12),
        # an O-grid from somebody else's generator: sides that halve only twice
        dict(name="steps_og181x91", kind="steps", form="ogrid", n0=181, n1=91, precision="fp64", steps=5),
        # the 513 x 513 configuration on the plain path
        dict(name="steps_og513", kind="steps", form="ogrid", n0=513, n1=513, precision="fp64", steps=5),
        # the 1025 x 1025 configuration in the precision form
        dict(name="steps_cav1025_mixed", kind="steps", form="cavity", n0=1025, n1=1025, precision="mixed", steps=5),
        # the benchmark: 256 O-grids of 65 .. 257 points a side in one batch
        dict(name="sweep256_og", kind="sweep", form="ogrid", ncases=256, sizes="sweep", precision="fp64", steps=8),
        # the converged-cases workload's form: cavities in the precision form
        dict(name="sweep64_cav_mixed", kind="sweep", form="cavity", ncases=64, sizes="sweep", precision="mixed", steps=8),
        # a parameter study: a handful of small cases of uneven size
        dict(name="ensemble12_og", kind="sweep", form="ogrid", ncases=12, sizes="small", precision="fp64", steps=10),
        # continuous batching: one slot of a running batch gets a new case, then a tick of steps
        dict(name="admit_tick_cav129", kind="admit", form="cavity", ncases=16, n0=129, n1=129, precision="mixed",
             steps=10),
        # a host program that owns the state: every step it goes up, one step runs, it comes back
        dict(name="hoststate64_og", kind="hoststate", form="ogrid", ncases=64, sizes="sweep", precision="fp64", steps=1),
        # gauss() of the reference replaced by the seam, at the reference's tolerance
        dict(name="gauss_og257", kind="gauss", form="ogrid", n0=257, n1=257, tol=SEAM_TOL),
        # sip9p() of the reference replaced by the seam
        dict(name="sip_cav257", kind="sip", form="cavity", n0=257, n1=257, tol=1e-6),
    ]


def _side(rng: random.Random, lo: int, hi: int, most: int) -> int:
    """A number of points near a log-uniform size: intervals = odd * 2^k, at most `most`
    intervals on the coarsest grid, so the sides halve unevenly often."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    k = 0
    while n / 2 ** k > most:
        k += 1
    return max(5, round(n / 2 ** k)) * 2 ** k + 1


def draw(rng: random.Random):
    kind = rng.choice(["timeloop", "steps", "steps", "sweep", "sweep", "admit", "hoststate", "gauss", "sip"])
    form = rng.choice(["ogrid", "cavity"])
    prec = rng.choice(["fp64", "mixed"])
    if kind in ("timeloop", "steps"):
        hi = 257 if kind == "timeloop" else 700
        return dict(kind=kind, form=form, n0=_side(rng, 33, hi, 40), n1=_side(rng, 33, hi, 40), precision=prec,
                    steps=rng.randint(3, 12))
    if kind in ("sweep", "hoststate"):
        return dict(kind=kind, form=form, ncases=int(round(math.exp(rng.uniform(math.log(4), math.log(100))))),
                    sizes=rng.choice(["sweep", "small"]), precision=prec,
                    steps=1 if kind == "hoststate" else rng.randint(3, 8))
    if kind == "admit":
        return dict(kind=kind, form=form, ncases=rng.randint(2, 32), n0=_side(rng, 65, 257, 40),
                    n1=_side(rng, 65, 257, 40), precision=prec, steps=rng.randint(5, 10))
    return dict(kind=kind, form=form, n0=_side(rng, 65, 1025, 40), n1=_side(rng, 65, 1025, 40),
                tol=rng.choice([SEAM_TOL, 1e-6]))


# ---- inputs -----------------------------------------------------------------
def _sizes(case):
    """(n0, n1) of every case; fixed by the case, not by the seed."""
    if case["kind"] not in ("sweep", "hoststate"):
        return [(case["n0"], case["n1"])] * case.get("ncases", 1)
    if case["sizes"] == "sweep":  # the benchmark's own sizes
        return [(d["N"], d["N"]) for d in sweep_draws(case["ncases"])]
    pick = [(33, 33), (49, 65), (65, 65), (65, 97), (97, 81), (129, 65)]
    return [pick[k % len(pick)] for k in range(case["ncases"])]


def _build(case, seed):
    sizes = _sizes(case)
    phys = sweep_draws(len(sizes), seed=int(seed) % (1 << 31))
    cfg = {65: "c1", 513: "c2", 1025: "c3"}.get(case.get("n0")) if len(sizes) == 1 else None
    grids, params = [], []
    prec = _lib.PRECISION_MIXED if case["precision"] == "mixed" else _lib.PRECISION_FP64
    for (n0, n1), d in zip(sizes, phys):
        if cfg:  # the single-case configurations keep their own Re, Ri, Pr; the skew is the seed's
            d = dict(CONFIGS[cfg], skew=d["skew"])
        if case["form"] == "ogrid":
            g = ogrid(n0, n1, ar=2.0, r_outer=20.0, skew=d["skew"])
            kw = dict(dt=1e-4, alpha=82.0)
        else:
            g = cavity(n0, n1, skew=d["skew"])
            kw = dict(dt=cavity_dt(max(n0, n1), d["Ri"], d["Re"], d["Pr"]))
        grids.append(g)
        params.append(case_params(g, Re=d["Re"], Ri=d["Ri"], Pr=d["Pr"], precision=prec, **kw))
    return grids, params, phys


def _host_image(batch):
    return torch.empty(batch.state_bytes() // 8, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("gauss", "sip"):
        return _prepare_seam(case, seed)
    grids, params, phys = _build(case, seed)
    st = dict(kind=kind, steps=case["steps"])
    if kind == "timeloop":
        p = params[0]
        s = Solver(grid=grids[0], Re=p.Re, Ri=p.Ri, Pr=p.Pr, dt=p.dt, alpha=p.alpha_deg, precision=p.precision)
        s.run_steps(4)
        st["solver"] = s
        return st
    b = Batch(grids, params)
    b.step(4)  # past the impulsive start, as a running program is
    st["batch"] = b
    st["image"] = _host_image(b)
    if kind == "admit":
        d = phys[0]
        st["new"] = (params[0], d["skew"], case["form"])
        st["slot"] = 0
        st["ncases"] = len(grids)
    if kind == "hoststate":
        b.get_state(st["image"])
    return st


# ---- one call -----------------------------------------------------------------
STATS = ("dmax", "cl", "cd", "cm", "nu", "circ", "q_l1", "q_l2", "dT_l1", "steady_res")


def _row(s):
    return [s[k] for k in STATS]


def run(st):
    kind = st["kind"]
    if kind == "gauss" or kind == "sip":
        return _run_seam(st)
    if kind == "timeloop":
        s = st["solver"]
        s.history.clear()
        s.timeLoop(st["steps"], write=False)
        out = s.fields()
        out["stats"] = np.array([_row(h) for h in s.history])
        return out
    b, image = st["batch"], st["image"]
    if kind == "admit":
        params, skew, form = st["new"]
        b.admit_spec(st["slot"], form, params, skew=skew)
        st["slot"] = (st["slot"] + 1) % st["ncases"]
        b.step(st["steps"])
        stats = b.all_stats()
        b.get_state(image)
        return {"state": image, "stats": np.array([_row(s) for s in stats])}
    if kind == "hoststate":
        b.set_state(image)
        b.step(st["steps"])
        b.get_state(image)
        return {"state": image, "stats": np.array(_row(b.stats(0)))}
    b.step(st["steps"])
    b.get_state(image)
    return {"state": image, "stats": np.array(_row(b.stats(0)))}


# ---- the two seams ---------------------------------------------------------------
GAUSS_OFFSETS = (  # (name, di, dj) in gauss()'s argument order
    ("p", 0, 0), ("e", 1, 0), ("s", 0, -1), ("n", 0, 1), ("w", -1, 0), ("se", 1, -1), ("sw", -1, -1), ("ne", 1, 1),
    ("nw", -1, 1), ("ss", 0, -2), ("ssee", 2, -2), ("ssww", -2, -2), ("sse", 1, -2), ("ssw", -1, -2), ("see", 2, -1),
    ("sww", -2, -1), ("nn", 0, 2), ("nnee", 2, 2), ("nnww", -2, 2), ("nne", 1, 2), ("nnw", -1, 2), ("nee", 2, 1),
    ("nww", -2, 1), ("ee", 2, 0), ("ww", -2, 0))
SIP_OFFSETS = (("p", 0, 0), ("e", 1, 0), ("s", 0, -1), ("n", 0, 1), ("w", -1, 0), ("se", 1, -1), ("sw", -1, -1),
               ("ne", 1, 1), ("nw", -1, 1))


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _momentum_planes(g, Re, dt):
    """The u system's coefficients (PSolver.cpp:765-882): 4th-order rows, 9-point near walls."""
    al, be, ga = (_cuda(x) for x in (g.alph, g.beta, g.gam))
    E, G, B = dt / Re * al / g.dxi0 ** 2, dt / Re * ga / g.dxi1 ** 2, dt / Re * be / (g.dxi0 * g.dxi1)
    near = torch.zeros((g.n1, g.n0), dtype=torch.bool, device="cuda")
    near[1] = near[g.n1 - 2] = True
    if g.kind == "cavity":
        near[:, 1] = near[:, g.n0 - 2] = True

    def rows(near_value, far_value):
        return torch.where(near, near_value, far_value)

    zero = torch.zeros_like(E)
    c = {"p": rows(1 + 2 * (E + G), 1 + 2.5 * (E + G))}
    for k in ("e", "w"):
        c[k] = rows(-E, -4.0 / 3.0 * E)
    for k in ("n", "s"):
        c[k] = rows(-G, -4.0 / 3.0 * G)
    for k in ("ne", "sw"):
        c[k] = rows(0.5 * B, 8.0 / 9.0 * B)
    for k in ("nw", "se"):
        c[k] = rows(-0.5 * B, -8.0 / 9.0 * B)
    for k, v in (("ee", E / 12), ("ww", E / 12), ("nn", G / 12), ("ss", G / 12), ("nnee", B / 72), ("ssww", B / 72),
                 ("nnww", -B / 72), ("ssee", -B / 72), ("nne", -B / 9), ("ssw", -B / 9), ("nee", -B / 9),
                 ("sww", -B / 9), ("nnw", B / 9), ("sse", B / 9), ("nww", B / 9), ("see", B / 9)):
        c[k] = rows(zero, v)
    if g.kind == "ogrid":  # wall rows are folded into the right-hand side
        for k in ("s", "se", "sw"):
            c[k][1] = 0.0
        for k in ("n", "ne", "nw"):
            c[k][g.n1 - 2] = 0.0
    return [c[name].contiguous() for name, _, _ in GAUSS_OFFSETS]


def _pressure_planes(g):
    """The pressure correction's 9-point coefficients (PSolver.cpp:944-1040)."""
    X, Y, E, G = (_cuda(a) for a in (g.xix, g.xiy, g.etx, g.ety))

    def at(a, di, dj):
        if g.kind == "ogrid" and di:  # unique columns wrap; the seam column repeats column 0
            u = torch.roll(a[:, :-1], -di, 1)
            a = torch.cat([u, u[:, :1]], 1)
        elif di:
            a = torch.roll(a, -di, 1)
        return torch.roll(a, -dj, 0) if dj else a

    c1, c2, c3 = 1 / (2 * g.dxi0 ** 2), 1 / (8 * g.dxi0 * g.dxi1), 1 / (2 * g.dxi1 ** 2)
    c = {k: torch.zeros_like(X) for k, _, _ in SIP_OFFSETS}
    for A, B in ((X, E), (Y, G)):
        e, w, n, s = at(A, 1, 0), at(A, -1, 0), at(A, 0, 1), at(A, 0, -1)
        be, bw, bn, bs = at(B, 1, 0), at(B, -1, 0), at(B, 0, 1), at(B, 0, -1)
        c["e"] += c1 * A * (A + e) + c2 * B * (n - s)
        c["w"] += c1 * A * (A + w) - c2 * B * (n - s)
        c["n"] += c2 * A * (be - bw) + c3 * B * (B + bn)
        c["s"] += -c2 * A * (be - bw) + c3 * B * (B + bs)
        c["ne"] += c2 * A * (B + be) + c2 * B * (A + n)
        c["sw"] += c2 * A * (B + bw) + c2 * B * (A + s)
        c["nw"] += -c2 * A * (B + bw) - c2 * B * (A + n)
        c["se"] += -c2 * A * (B + be) - c2 * B * (A + s)
        c["p"] += -c1 * A * (2 * A + w + e) - c3 * B * (2 * B + bs + bn)
    return [c[name].contiguous() for name, _, _ in SIP_OFFSETS]


def _apply(planes, offsets, phi, periodic):
    """A phi on the unknown cells (zero elsewhere); `phi` holds the boundary values."""
    n1, n0 = phi.shape
    P = n0 - 1 if periodic else n0
    core = phi[:, :P]
    out = torch.zeros_like(core)
    for a, (_, di, dj) in zip(planes, offsets):
        out += a[:, :P] * torch.roll(core, (-dj, -di), (0, 1))
    full = torch.cat([out, out[:, :1]], 1) if periodic else out
    full[0] = full[-1] = 0.0
    if not periodic:
        full[:, 0] = full[:, -1] = 0.0
    return full


def _fields(case, seed):
    """(grid, physics, the system's solution, its first guess) of a seam case."""
    d = sweep_draws(1, seed=int(seed) % (1 << 31))[0]
    n0, n1 = case["n0"], case["n1"]
    g = ogrid(n0, n1, ar=2.0, r_outer=20.0, skew=d["skew"]) if case["form"] == "ogrid" else cavity(n0, n1, skew=d["skew"])
    gen = np.random.default_rng(int(seed))
    XI, ETA = np.meshgrid(np.arange(n0) / (n0 - 1), np.arange(n1) / (n1 - 1))

    def smooth(modes, scale):
        f = np.zeros((n1, n0))
        for _ in range(modes):
            kx, ky = gen.integers(1, 7, size=2)
            f += scale * gen.standard_normal() * np.cos(2 * math.pi * (kx * XI + gen.random())) * np.sin(math.pi * ky * ETA)
        if g.kind == "ogrid":
            f[:, -1] = f[:, 0]
        else:
            f *= np.sin(math.pi * XI)
        return f

    if case["kind"] == "sip":  # a pressure correction: zero boundary values, zero first guess
        return g, d, smooth(8, 1.0), np.zeros((n1, n0))
    first = 1.0 + smooth(8, 0.3)  # a velocity component, and what one step changes in it
    return g, d, first + smooth(8, 1e-3), first


def _prepare_seam(case, seed):
    g, d, true, first = _fields(case, seed)
    periodic = int(g.kind == "ogrid")
    if case["kind"] == "gauss":
        dt = 1e-4 if periodic else cavity_dt(max(g.n0, g.n1), d["Ri"], d["Re"], d["Pr"])
        planes, offsets = _momentum_planes(g, d["Re"], dt), GAUSS_OFFSETS
    else:
        planes, offsets = _pressure_planes(g), SIP_OFFSETS
    q = _apply(planes, offsets, _cuda(true), periodic)
    return dict(kind=case["kind"], planes=planes, ptrs=(ctypes.c_void_p * len(planes))(*[p.data_ptr() for p in planes]),
                first=_cuda(first), phi=torch.empty_like(q), q=q, n0=g.n0, n1=g.n1, periodic=periodic,
                tol=case["tol"])


def _run_seam(st):
    L = _lib.lib()
    st["phi"].copy_(st["first"])
    count = ctypes.c_int(0)
    fn = L.cfd_gauss_solve if st["kind"] == "gauss" else L.cfd_sip_solve
    _lib.check(fn(st["n0"], st["n1"], st["periodic"], st["ptrs"], ctypes.c_void_p(st["phi"].data_ptr()),
                  ctypes.c_void_p(st["q"].data_ptr()), st["tol"], 100000, ctypes.byref(count), None), st["kind"])
    return {"phi": st["phi"], "iterations": count.value}


# ---- what a call cannot do without -------------------------------------------------
STEP_PLANES = 19    # u, v, p, T, up, vp read and written, seven metrics read
STEP_FLOPS = 700    # per cell: convection and sources, two sweeps of five systems, one preconditioned iteration


def work(case):
    if case["kind"] in ("gauss", "sip"):
        cells = case["n0"] * case["n1"]
        planes = (25 if case["kind"] == "gauss" else 9) + 3
        return {"bytes": 8.0 * planes * cells, "flops": 2.0 * planes * cells}
    cells = sum(n0 * n1 for n0, n1 in _sizes(case))
    return {"bytes": 8.0 * STEP_PLANES * cells * case["steps"], "flops": float(STEP_FLOPS) * cells * case["steps"]}


def exact(case, seed):
    """The seams' systems are made from their solution. A time step has no such value: its
    inner solves stop at a tolerance."""
    if case["kind"] not in ("gauss", "sip"):
        return None
    return {"phi": torch.from_numpy(_fields(case, seed)[2]), "iterations": None}
