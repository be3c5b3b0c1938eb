"""Performance cases of the framework: the calls its users make, over the sizes they make them at.

Every case goes through the public entry points (``TGVSolver``, ``Ensemble``, ``FullSolver``, the
line operators, ``final_kinetic_energy``, and the C ABI's device upload and download, which the
Python classes leave to the caller). ``exact`` restates each of them in torch FP64 on dense operator
matrices, independently of the library.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import astr_gpu_b200 as ag
from astr_gpu_b200.adjoint import final_kinetic_energy

HM = 5                       # halo nodes on each side of a line
ALFA, BETA_HALO, GAMMA = 0.49, 1.11, 1.4
PRANDTL, REF_TEM = 0.72, 273.15
RK = ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0))

# ---------------------------------------------------------------------------------------- cases


def listed():
    return [
        # RK3 steps of the periodic box with the state in device memory. The smallest box users
        # step (the ensemble's smallest), several steps per call: launch latency.
        dict(name="step_32", kind="step", im=32, jm=32, km=32, nsteps=4, filter=True, mach=0.1, reynolds=1600.0),
        # a box with three different sizes, two of them odd, filter off (a resolved run)
        dict(name="step_odd", kind="step", im=83, jm=50, km=65, nsteps=2, filter=False, mach=0.3, reynolds=400.0),
        # the grid of the reference's committed Taylor-Green history
        dict(name="step_128", kind="step", im=128, jm=128, km=128, nsteps=2, filter=True, mach=0.1, reynolds=1600.0),
        # the headline Taylor-Green box
        dict(name="step_512", kind="step", im=512, jm=512, km=512, nsteps=1, filter=True, mach=0.1, reynolds=1600.0),
        # one step of a Fortran caller whose state lives in host memory
        dict(name="host_128", kind="host", im=128, jm=128, km=128, nsteps=1, filter=True, mach=0.1, reynolds=1600.0),
        # independent boxes of uneven sizes advanced together
        dict(name="ensemble_12", kind="ensemble", boxes="32,32,32,48,48,48,64,64,64,96,96,128", nsteps=2, mach=0.3,
             reynolds=1600.0),
        # gradients of a velocity field along the three axes: the reference's gradient kernel test
        dict(name="gradient_256", kind="lines", op="central", im=256, jm=256, km=256, nf=3, ntype="3,3,3"),
        # filterq of a channel's conserved variables: walls along y, odd sizes
        dict(name="filter_walls", kind="lines", op="filter", im=150, jm=97, km=75, nf=5, ntype="3,4,3"),
        # the upwind and downwind interface flux of one small block, one physical end
        dict(name="flux_small", kind="lines", op="flux", im=40, jm=33, km=32, nf=1, ntype="3,1,2"),
        # the full solver's step: a channel with no-slip walls, central convection
        dict(name="full_channel", kind="full", im=128, jm=97, km=96, nsteps=1, ntype="3,4,3", conschm=643, bfac=0.0,
             char=False, shkcrt=0.01, mach=0.3, reynolds=400.0),
        # the reference's compressible example set-up: upwind compact flux in characteristic
        # variables with the shock sensor
        dict(name="full_upwind", kind="full", im=96, jm=96, km=96, nsteps=1, ntype="3,3,3", conschm=543, bfac=0.3,
             char=True, shkcrt=0.001, mach=0.5, reynolds=1600.0),
        # gradient of the final kinetic energy through a few steps (forward and backward)
        dict(name="adjoint_64", kind="adjoint", im=64, jm=64, km=64, nsteps=4, every=2, filter=True, mach=0.3,
             reynolds=180.0),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, points):
    while True:
        n = [_size(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= points:
            return dict(im=n[0], jm=n[1], km=n[2])


def draw(rng):
    kind = rng.choice(["step", "step", "step", "host", "ensemble", "lines", "lines", "full", "full", "adjoint"])
    mach, reynolds = round(rng.uniform(0.1, 0.5), 3), round(math.exp(rng.uniform(math.log(200), math.log(3000))), 1)
    if kind == "step":
        return dict(kind=kind, **_box(rng, 24, 400, 4e7), nsteps=rng.randint(1, 3), filter=rng.random() < 0.75, mach=mach,
                    reynolds=reynolds)
    if kind == "host":
        return dict(kind=kind, **_box(rng, 24, 200, 4e6), nsteps=rng.randint(1, 2), filter=True, mach=mach,
                    reynolds=reynolds)
    if kind == "ensemble":
        sizes = sorted(_size(rng, 24, 128) for _ in range(rng.randint(3, 14)))
        return dict(kind=kind, boxes=",".join(map(str, sizes)), nsteps=rng.randint(1, 3), mach=mach, reynolds=reynolds)
    if kind == "lines":
        nt = ",".join(str(rng.choice([3, 3, 1, 2, 4])) for _ in range(3))
        return dict(kind=kind, op=rng.choice(["central", "filter", "flux", "fluxdiff"]), **_box(rng, 24, 600, 2e7),
                    nf=rng.randint(1, 5), ntype=nt)
    if kind == "full":
        char = rng.random() < 0.4
        conschm = 543 if char or rng.random() < 0.3 else 643
        nt = "3,3,3" if conschm == 543 else rng.choice(["3,3,3", "3,4,3", "4,3,3", "3,3,4"])
        return dict(kind=kind, **_box(rng, 24, 160, 1.5e6), nsteps=1, ntype=nt, conschm=conschm,
                    bfac=round(rng.uniform(0.1, 0.7), 2) if conschm == 543 else 0.0, char=char, shkcrt=0.001, mach=mach,
                    reynolds=reynolds)
    return dict(kind=kind, **_box(rng, 24, 80, 3e5), nsteps=rng.randint(2, 5), every=rng.randint(1, 4), filter=True,
                mach=mach, reynolds=reynolds)


# --------------------------------------------------------------------------------------- inputs


def _dims(case):
    return case["im"], case["jm"], case["km"]


def _ints(text):
    return [int(x) for x in str(text).split(",")]


def _flow(n, seed, mach, walls=(False, False, False)):
    """q(0..N, 5) of a Taylor-Green field with four random modes on top, as a (5, k, j, i) CUDA
    tensor (its bytes are the Fortran array q(i, j, k, 5)); the velocity vanishes on walls."""
    rnd = np.random.RandomState(seed % (1 << 32))
    ax = []
    for d in range(3):
        i = torch.arange(n[d] + 1, device="cuda", dtype=torch.float64)
        if not walls[d]:
            i = torch.remainder(i, float(n[d]))
        ax.append((i * (2.0 * math.pi / n[d])).view([-1 if 2 - d == a else 1 for a in range(3)]))
    x, y, z = ax
    shape = (n[2] + 1, n[1] + 1, n[0] + 1)
    q = torch.empty((5,) + shape, dtype=torch.float64, device="cuda")
    q[1] = torch.sin(x) * torch.cos(y) * torch.cos(z)
    q[2] = -torch.cos(x) * torch.sin(y) * torch.cos(z)
    q[3] = 0.0
    for _ in range(4):
        k = rnd.randint(1, 5, 3) * rnd.choice([-1, 1], 3)
        wave = torch.cos(float(k[0]) * x + float(k[1]) * y + float(k[2]) * z + rnd.uniform(0, 2 * math.pi))
        for c, a in enumerate(rnd.normal(0.0, 0.08, 3)):
            q[1 + c].add_(wave, alpha=float(a))
        del wave
    for d in range(3):
        if walls[d]:
            q[1:4] *= torch.sin(0.5 * ax[d])
    p = 1.0 / (GAMMA * mach * mach) + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
    q[0] = p * (GAMMA * mach * mach)                 # temperature 1
    q[4] = p / (GAMMA - 1.0)
    del p
    for c in range(3):
        q[4] += 0.5 * q[0] * q[1 + c] ** 2
    for c in range(3):
        q[1 + c] *= q[0]
    return q


def _dt(n, mach):
    """About CFL 0.5 for these fields (|u| up to about 1.5, sound speed 1/M)."""
    return 0.5 / ((1.5 + 1.0 / mach) * sum(m / (2.0 * math.pi) for m in n))


def _field(n, nf, seed):
    """nf smooth-plus-noise fields on nodes -5..N+5 of every axis (interpolated turbulence data has
    content at every wavenumber), as a (nf, k, j, i) CUDA tensor."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = tuple(m + 1 + 2 * HM for m in reversed(n))
    f = 0.1 * torch.randn((nf,) + shape, generator=g, dtype=torch.float64, device="cuda")
    ax = [torch.arange(-HM, m + HM + 1, device="cuda", dtype=torch.float64) * (2 * math.pi / m) for m in n]
    base = torch.cos(ax[2]).view(-1, 1, 1) * torch.sin(2 * ax[1]).view(1, -1, 1) * torch.cos(3 * ax[0]).view(1, 1, -1)
    return f + base


def _fortran(t):
    """The (i, j, k[, m]) Fortran-ordered view of a (m, k, j, i) or (k, j, i) tensor."""
    return t.permute(*reversed(range(t.dim())))


def _i64(v):
    return (ctypes.c_int64 * 3)(*[int(x) for x in v])


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _params(case, sutherland=110.4):
    extra = {}
    if case["kind"] == "full":
        extra = dict(ntype=tuple(_ints(case["ntype"])), conschm=case["conschm"], bfacmpld=case["bfac"],
                     lchardecomp=case["char"], shkcrt=case["shkcrt"])
    return ag.FlowParams(mach=case["mach"], reynolds=case["reynolds"], sutherland=sutherland,
                         filter_on=case.get("filter", True), **extra)


class _Context:
    """One library context per process, as a user's program has."""
    ctx = None

    @classmethod
    def get(cls):
        if cls.ctx is None:
            cls.ctx = ag.Context(0)
        return cls.ctx


def prepare(case, seed):
    ctx = _Context.get()
    kind = case["kind"]
    if kind == "ensemble":
        sizes = _ints(case["boxes"])
        boxes = [ag.TGVSolver(ctx, m, params=_params(case)) for m in sizes]
        q = [_flow((m,) * 3, seed * 64 + b, case["mach"]) for b, m in enumerate(sizes)]
        return dict(case=case, ens=ag.Ensemble(ctx, boxes), boxes=boxes, q=q, out=[torch.empty_like(x) for x in q],
                    dt=[_dt((m,) * 3, case["mach"]) for m in sizes])
    n = _dims(case)
    if kind == "lines":
        nt = _ints(case["ntype"])
        if case["op"] == "central":
            sch = [[ag.fd_scheme_initiate(ctx, "643c", nt[d], n[d])] for d in range(3)]
        elif case["op"] == "filter":
            sch = [[ag.compact_filter_initiate(ctx, nt[d], n[d])] for d in range(3)]
        else:
            sch = [[ag.compact_flux_initiate(ctx, nt[d], n[d], w, 0.3) for w in "+-"] for d in range(3)]
        return dict(case=case, ctx=ctx, schemes=sch, f=_fortran(_field(n, case["nf"], seed)))
    walls = tuple(t != 3 for t in _ints(case.get("ntype", "3,3,3")))
    q = _flow(n, seed, case["mach"], walls)
    state = dict(case=case, ctx=ctx, q=q, dt=_dt(n, case["mach"]), shape=[m + 1 for m in n])
    if kind == "full":
        state["solver"] = ag.FullSolver(ctx, *n, params=_params(case, 110.3))
        state["out"] = torch.empty_like(q)
        return state
    state["solver"] = ag.TGVSolver(ctx, *n, params=_params(case))
    if kind == "step":
        state["out"] = torch.empty_like(q)
    elif kind == "host":
        state["q"] = np.asfortranarray(_fortran(q).cpu().numpy())
    else:
        state["q"] = _fortran(q)
    return state


# ------------------------------------------------------------------------------------- one pass


def _upload(ctx, call, solver, q):
    shape = [m for m in reversed(q.shape[1:])]
    ctx.check(call(solver._h, _ptr(q), _i64(shape), _i64((0, 0, 0)), ag.ASTR_DEVICE))


_download = _upload   # the same arguments


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        ctx = state["ens"].ctx
        for b, q in zip(state["boxes"], state["q"]):
            _upload(ctx, ctx.L.astr_state_upload, b, q)
        state["ens"].step(state["dt"], case["nsteps"])
        for b, out in zip(state["boxes"], state["out"]):
            _download(ctx, ctx.L.astr_state_download, b, out)
        return [list(out) for out in state["out"]]
    ctx = state["ctx"]
    if kind == "lines":
        n, f, nf = _dims(case), state["f"], case["nf"]
        call = {"central": ag.central, "filter": ag.compact_filter, "flux": ag.flux_compact,
                "fluxdiff": ag.flux_difference}[case["op"]]
        outs = []
        for d in range(3):
            lo = [0, 0, 0]
            ext = [m + 1 for m in n]
            if case["op"] == "flux":
                lo[d], ext[d] = -1, n[d] + 2
            scale = {} if case["op"] in ("filter", "flux") else {"scale": n[d] / (2 * math.pi)}
            for s in state["schemes"][d]:
                outs.append(call(ctx, s, f, d, lbound=(-HM,) * 3, out_lbound=lo, out_shape=ext, **scale))
        return outs
    solver, q = state["solver"], state["q"]
    if kind == "host":
        diag = solver.rk3_host(q, state["dt"], case["nsteps"])
        return [q[..., m] for m in range(5)] + [diag]
    if kind == "adjoint":
        q0 = q.detach().requires_grad_(True)
        J = final_kinetic_energy(q0, solver, state["dt"], case["nsteps"], case["every"])
        J.backward()
        return [J.detach()] + [q0.grad[..., m] for m in range(5)]
    if kind == "full":
        _upload(ctx, ctx.L.astr_full_upload, solver, q)
        solver.step(state["dt"], case["nsteps"])
        _download(ctx, ctx.L.astr_full_download, solver, state["out"])
    else:
        _upload(ctx, ctx.L.astr_state_upload, solver, q)
        solver.rk3(state["dt"], case["nsteps"])
        _download(ctx, ctx.L.astr_state_download, solver, state["out"])
    return list(state["out"])


# Operations of one stage per node: 27 derivative and 15 filter line solves (right-hand side, two
# sweeps), the gradients' and fluxes' pointwise work.
STAGE_FLOPS = 27 * 11 + 15 * 20 + 200


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        points = sum((m + 1) ** 3 for m in _ints(case["boxes"]))
    else:
        points = math.prod(m + 1 for m in _dims(case))
    if kind == "lines":
        per = {"central": 11, "filter": 20, "flux": 14, "fluxdiff": 14}[case["op"]]
        winds = 2 if case["op"].startswith("flux") else 1
        return dict(bytes=8.0 * case["nf"] * points * (1 + 3 * winds), flops=float(per * 3 * winds * case["nf"] * points))
    steps = case["nsteps"]
    flops = 3.0 * steps * STAGE_FLOPS * points
    if kind == "adjoint":
        return dict(bytes=80.0 * points * steps * 2, flops=3.0 * flops)
    if kind == "full" and case["conschm"] == 543:
        flops += 3.0 * steps * points * (15 * 60 + (3 * 600 if case["char"] else 0))
    return dict(bytes=80.0 * points * steps, flops=flops)


def tolerance(case):
    """About four times the difference from ``exact`` at the same precision (FP64 throughout)."""
    kind = case["kind"]
    if kind == "lines":     # the filter's systems are nearly singular (alpha 0.49): ten times the others
        return {"rel": 1.6e-14, "max": 1e-12} if case["op"] == "filter" else {"rel": 2e-15, "max": 1e-13}
    if kind == "full" and case["conschm"] == 543:   # the limiter branches at an absolute 1e-10
        return {"rel": 4e-13, "max": 1e-8}
    return {"rel": 4e-13, "max": 4e-11}


# ------------------------------------------------------------------------------------- restated
# Line operators as dense matrices over the line's nodes -5..N+5 (derivative.F90, filter.F90,
# flux.F90): rows of R A^-1 B for the output nodes.


def _solve(a, c, B):
    A = np.eye(len(a)) + np.diag(a[1:], -1) + np.diag(c[:-1], 1)
    return np.linalg.solve(A, B)


def _deriv_matrix(n, nt):
    lp, rp = nt in (1, 4), nt in (2, 4)
    first, last = (0 if lp else -1), (n if rp else n + 1)
    rows = last - first + 1
    B = np.zeros((rows, n + 1 + 2 * HM))
    a, c = np.full(rows, 1.0 / 3.0), np.full(rows, 1.0 / 3.0)

    def put(r, terms):
        for off, w in terms.items():
            B[r, first + r + off + HM] += w

    for r in range(2 if lp else 1, rows - (2 if rp else 1)):
        put(r, {1: 7 / 9, -1: -7 / 9, 2: 1 / 36, -2: -1 / 36})
    six = {1: 0.75, -1: -0.75, 2: -0.15, -2: 0.15, 3: 1 / 60, -3: -1 / 60}
    a[0] = c[0] = a[-1] = c[-1] = 0.0
    if lp:
        a[0] = c[0] = 2.0
        a[1] = c[1] = 0.25
        put(0, {0: -2.5, 1: 2.0, 2: 0.5})
        put(1, {1: 0.75, -1: -0.75})
    else:
        put(0, six)
    if rp:
        a[-1] = c[-1] = 2.0
        a[-2] = c[-2] = 0.25
        put(rows - 1, {0: 2.5, -1: -2.0, -2: -0.5})
        put(rows - 2, {1: 0.75, -1: -0.75})
    else:
        put(rows - 1, six)
    return _solve(a, c, B)[-first:-first + n + 1]


def _filter_matrix(n, nt, bb):
    lp, rp = nt in (1, 4), nt in (2, 4)
    first, last = (0 if lp else -3), (n if rp else n + 3)
    rows = last - first + 1
    al = ALFA
    B = np.zeros((rows, n + 1 + 2 * HM))
    a, c = np.full(rows, al), np.full(rows, al)
    a[0] = c[0] = 0.98 if lp else BETA_HALO
    a[-1] = c[-1] = 0.98 if rp else BETA_HALO
    c6 = [(11 + 10 * al) / 32, (15 + 34 * al) / 64, (-3 + 6 * al) / 32, (1 - 2 * al) / 64]
    c8 = [(93 + 70 * al) / 256, (7 + 18 * al) / 32, (-7 + 14 * al) / 64, (1 - 2 * al) / 32, (-1 + 2 * al) / 256]
    c10 = [(193 + 126 * al) / 512, (105 + 302 * al) / 512, (-15 + 30 * al) / 128, (45 - 90 * al) / 1024,
           (-5 + 10 * al) / 512, (1 - 2 * al) / 1024]
    onesided = [
        [(63 + bb) / 64, (3 + 29 * bb) / 32, (-15 + 15 * bb) / 64, (5 - 5 * bb) / 16, (-15 + 15 * bb) / 64,
         (3 - 3 * bb) / 32, (-1 + bb) / 64],
        [(1 + 62 * al) / 64, (29 + 6 * al) / 32, (15 + 34 * al) / 64, (-5 + 10 * al) / 16, (15 - 30 * al) / 64,
         (-3 + 6 * al) / 32, (1 - 2 * al) / 64],
        [(-1 + 2 * al) / 64, (3 + 26 * al) / 32, (49 + 30 * al) / 64, (5 + 6 * al) / 16, (-15 + 30 * al) / 64,
         (3 - 6 * al) / 32, (-1 + 2 * al) / 64]]
    bh = BETA_HALO
    halo = [
        [(-1 + bh) / 1024, (5 - 5 * bh) / 512, (979 + 45 * bh) / 1024, (15 + 113 * bh) / 128, (-105 + 105 * bh) / 512,
         (63 - 63 * bh) / 256, (-105 + 105 * bh) / 512, (15 - 15 * bh) / 128, (-45 + 45 * bh) / 1024,
         (5 - 5 * bh) / 512, (-1 + bh) / 1024],
        [(1 - 2 * al) / 1024, (-5 + 10 * al) / 512, (45 + 934 * al) / 1024, (113 + 30 * al) / 128,
         (105 + 302 * al) / 512, (-63 + 126 * al) / 256, (105 - 210 * al) / 512, (-15 + 30 * al) / 128,
         (45 - 90 * al) / 1024, (-5 + 10 * al) / 512, (1 - 2 * al) / 1024],
        [(-1 + 2 * al) / 1024, (5 - 10 * al) / 512, (-45 + 90 * al) / 1024, (15 + 98 * al) / 128,
         (407 + 210 * al) / 512, (63 + 130 * al) / 256, (-105 + 210 * al) / 512, (15 - 30 * al) / 128,
         (-45 + 90 * al) / 1024, (5 - 10 * al) / 512, (-1 + 2 * al) / 1024]]

    def symmetric(r, w):
        for k, v in enumerate(w):
            B[r, first + r + HM + k] += v
            B[r, first + r + HM - k] += v

    for end, phys in ((0, lp), (1, rp)):
        for k in range(5 if phys else 3):
            r = k if end == 0 else rows - 1 - k
            sgn, base = (1, first) if end == 0 else (-1, last)
            if not phys:
                for j in range(11):
                    B[r, base + sgn * (j - 2) + HM] += halo[k][j]
            elif k < 3:
                for j in range(7):
                    B[r, base + sgn * j + HM] += onesided[k][j]
            else:
                symmetric(r, c6 if k == 3 else c8)
    for r in range(5 if lp else 3, rows - (5 if rp else 3)):
        symmetric(r, c10)
    M = _solve(a, c, B)[-first:-first + n + 1]
    for end, phys in ((0, lp), (n, rp)):             # the boundary node is reset to its input
        if phys:
            M[end] = 0.0
            M[end, end + HM] = 1.0
    return M


def _flux_matrix(n, nt, wind, b):
    lp, rp = nt in (1, 4), nt in (2, 4)
    first, last = (-1 if lp else -2), (n if rp else n + 1)
    rows = last - first + 1
    B = np.zeros((rows, n + 1 + 2 * HM))
    lo, hi = 0.5 - b / 6.0, 1.0 / 6.0 + b / 6.0
    a, c = np.full(rows, lo if wind == "+" else hi), np.full(rows, hi if wind == "+" else lo)
    w = [1 / 18 - b / 36, 19 / 18 - 9 * b / 36, 5 / 9 + 9 * b / 36, b / 36]

    def put(r, terms):
        for off, v in terms.items():
            B[r, first + r + off + HM] += v

    for r in range(2 if lp else 1, rows - (2 if rp else 1)):
        put(r, {k - 1 if wind == "+" else 2 - k: w[k] for k in range(4)})
    six = {0: 37 / 60, 1: 37 / 60, -1: -2 / 15, 2: -2 / 15, -2: 1 / 60, 3: 1 / 60}
    a[0] = c[0] = a[-1] = c[-1] = 0.0
    if lp:
        a[0] = c[0] = 2.0
        a[1] = c[1] = 0.25
        put(0, {1: 2.5, 2: 0.5})
        put(1, {0: 0.75, 1: 0.75})
    else:
        put(0, six)
    if rp:
        a[-1] = c[-1] = 2.0
        a[-2] = c[-2] = 0.25
        put(rows - 1, {0: 2.5, -1: 0.5})
        put(rows - 2, {1: 0.75, 0: 0.75})
    else:
        put(rows - 1, six)
    return _solve(a, c, B)[-1 - first:-1 - first + n + 2]


def _periodic(M, n):
    """The operator over nodes 0..N of a periodic line: f(-k) = f(N-k), f(N+k) = f(k)."""
    P = np.zeros((M.shape[0], n + 1))
    for t in range(-HM, n + HM + 1):
        P[:, t + n if t < 0 else (t - n if t > n else t)] += M[:, t + HM]
    return P


def _cuda(M):
    return torch.from_numpy(np.ascontiguousarray(M)).cuda()


def _along(M, f, d):
    """M applied along direction d (0 x, 1 y, 2 z) of a (k, j, i) field."""
    if d == 0:
        return f @ M.T
    if d == 1:
        return torch.matmul(M, f)
    return (M @ f.reshape(f.shape[0], -1)).reshape((M.shape[0],) + tuple(f.shape[1:]))


class _Thermo:
    def __init__(self, case, sutherland):
        m = case["mach"]
        self.c2, self.c5, self.c6 = GAMMA * m * m, (GAMMA - 1) * m * m, 1.0 / (GAMMA - 1)
        self.tc, self.re, self.mach = sutherland / REF_TEM, case["reynolds"], m

    def prims(self, q):
        u = [q[1 + c] / q[0] for c in range(3)]
        p = (q[4] - 0.5 * q[0] * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])) / self.c6
        return u, p, p / q[0] * self.c2

    def viscous(self, G, GT, u, T):
        """sigma[a][b] and the heat and work flux from G[a][d] = du_a/dx_d and GT[d]."""
        s = [[0.5 * (G[a][b] + G[b][a]) for b in range(3)] for a in range(3)]
        skk = (s[0][0] + s[1][1] + s[2][2]) / 3.0
        miu = T * torch.sqrt(T) * (1.0 + self.tc) / (T + self.tc) / self.re
        sig = [[2.0 * miu * (s[a][b] - skk if a == b else s[a][b]) for b in range(3)] for a in range(3)]
        hcc = miu / PRANDTL / self.c5
        return sig, [hcc * GT[d] + sig[d][0] * u[0] + sig[d][1] * u[1] + sig[d][2] * u[2] for d in range(3)]


class _BoxStep:
    """The periodic box's RK3 step: rhscal, update, filter."""

    def __init__(self, n, case):
        self.th = _Thermo(case, 110.4)
        self.filter_on = case.get("filter", True)
        self.D = [_cuda(_periodic(_deriv_matrix(m, 3), m) * (m / (2 * math.pi))) for m in n]
        self.F = [_cuda(_periodic(_filter_matrix(m, 3, 1.09), m)) for m in n]

    def rhs(self, q):
        th, D = self.th, self.D
        u, p, T = th.prims(q)
        G = [[_along(D[d], u[a], d) for d in range(3)] for a in range(3)]
        GT = [_along(D[d], T, d) for d in range(3)]
        sig, qf = th.viscous(G, GT, u, T)
        del G, GT, T
        R = [0.0] * 5
        for d in range(3):
            for m in range(5):
                if m == 0:
                    f = -q[1 + d]
                elif m < 4:
                    f = sig[d][m - 1] - q[m] * u[d]
                    f = f - p if m - 1 == d else f
                else:
                    f = qf[d] - (q[4] + p) * u[d]
                R[m] = R[m] + _along(D[d], f, d)
        return R

    def step(self, q, dt):
        q = list(q)
        start = q
        for c1, c2, c3 in RK:
            R = self.rhs(q)
            q = [c1 * start[m] + c2 * q[m] + c3 * dt * R[m] for m in range(5)]
            del R
            if self.filter_on:
                for d in range(3):
                    q = [_along(self.F[d], x, d) for x in q]
        return q

    def diagnostics(self, q):
        """Kinetic energy, enstrophy and dissipation over nodes 1..N."""
        th = self.th
        u, _, T = th.prims(q)
        G = [[_along(self.D[d], u[a], d) for d in range(3)] for a in range(3)]
        om = [G[2][1] - G[1][2], G[0][2] - G[2][0], G[1][0] - G[0][1]]
        s = [[0.5 * (G[a][b] + G[b][a]) for b in range(3)] for a in range(3)]
        div = s[0][0] + s[1][1] + s[2][2]
        miu = T * torch.sqrt(T) * (1.0 + th.tc) / (T + th.tc) / th.re
        ss = sum(s[a][b] ** 2 for a in range(3) for b in range(3))
        mean = lambda x: float(x[1:, 1:, 1:].mean())  # noqa: E731
        return np.array([0.5 * mean(q[0] * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)),
                         0.5 * mean(q[0] * (om[0] ** 2 + om[1] ** 2 + om[2] ** 2)),
                         mean(2.0 * miu * (ss - div * div / 3.0))])


def _minmod(*v):
    lo = torch.stack([x.abs() for x in v]).amin(0)
    pos = torch.stack([x > 0 for x in v]).all(0)
    neg = torch.stack([x < 0 for x in v]).all(0)
    return torch.where(pos, lo, torch.where(neg, -lo, torch.zeros_like(lo)))


def _mp5(u, ul, shock):
    ump = u[2] + _minmod(u[3] - u[2], 4.0 * (u[2] - u[1]))
    active = shock & ((ul - u[2]) * (ul - ump) >= 1.0e-10)
    dm1, d0, d1 = u[0] - 2 * u[1] + u[2], u[1] - 2 * u[2] + u[3], u[2] - 2 * u[3] + u[4]
    dhm1 = _minmod(4 * dm1 - d0, 4 * d0 - dm1, dm1, d0)
    dh0 = _minmod(4 * d0 - d1, 4 * d1 - d0, d0, d1)
    uul = u[2] + 4.0 * (u[2] - u[1])
    umd = 0.5 * (u[2] + u[3]) - 0.5 * dh0
    ulc = u[2] + 0.5 * (u[2] - u[1]) + 1.333333333333333 * dhm1
    mn, mx = torch.minimum, torch.maximum
    umin = mx(mn(mn(u[2], u[3]), umd), mn(mn(u[2], uul), ulc))
    umax = mn(mx(mx(u[2], u[3]), umd), mx(mx(u[2], uul), ulc))
    return torch.where(active, ul + _minmod(umin - ul, umax - ul), ul)


class _FullStep:
    """The full solver's stage: filter, walls, qswap, rhscal in metric form, update, primitives.
    Halos of a direction hold what qswap saw when it copied them."""

    def __init__(self, n, case):
        self.n, self.case, self.th = n, case, _Thermo(case, 110.3)
        self.nt = _ints(case["ntype"])
        self.rd = [m / (2 * math.pi) for m in n]
        self.jac = math.prod(2 * math.pi / m for m in n)
        self.D = [_cuda(_deriv_matrix(m, t)) for m, t in zip(n, self.nt)]
        F = [_filter_matrix(m, t, 1.09) for m, t in zip(n, self.nt)]
        self.F = [_cuda(_periodic(M, m) if t == 3 else M[:, HM:HM + m + 1]) for M, m, t in zip(F, n, self.nt)]
        if case["conschm"] == 543:
            self.W = [[_cuda(_flux_matrix(m, t, w, case["bfac"])) for w in "+-"] for m, t in zip(n, self.nt)]

    def cut(self, f, d, lo, hi):
        """Nodes lo..hi-1 of f along d."""
        return f.narrow(2 - d, lo, hi - lo)

    def wrap(self, f, d):
        """f with its periodic images (zeros past physical ends, which no operator reads)."""
        n = self.n[d]
        lo, hi = self.cut(f, d, n - HM, n), self.cut(f, d, 1, HM + 1)
        if self.nt[d] != 3:
            lo, hi = torch.zeros_like(lo), torch.zeros_like(hi)
        return torch.cat([lo, f, hi], 2 - d)

    def walls(self, q, pr):
        th = self.th
        for d in range(3):
            for side, has in ((0, self.nt[d] in (1, 4)), (1, self.nt[d] in (2, 4))):
                if not has:
                    continue
                at = [0, 1, 2] if side == 0 else [self.n[d] - k for k in range(3)]
                p1, p2 = (pr[4].select(2 - d, k) for k in at[1:])
                pe = (4.0 * p1 - p2) / 3.0
                for c in (1, 2, 3):
                    pr[c].select(2 - d, at[0]).zero_()
                    q[c].select(2 - d, at[0]).zero_()
                pr[4].select(2 - d, at[0]).copy_(pe)
                pr[5].select(2 - d, at[0]).fill_(1.0)
                for f in (pr[0], q[0]):
                    f.select(2 - d, at[0]).copy_(pe * th.c2)
                q[4].select(2 - d, at[0]).copy_(pe * th.c6)

    def primitives(self, q):
        u, p, T = self.th.prims(q)
        return [q[0].clone(), *u, p, T]

    def swap(self, q, pr):
        """Halo values (q, primitives) per periodic direction; planes 0 and N averaged."""
        halos = {}
        for d in range(3):
            if self.nt[d] != 3:
                continue
            n = self.n[d]
            lo = [self.cut(f, d, n - HM, n).clone() for f in q]
            hi = [self.cut(f, d, 1, HM + 1).clone() for f in q]
            for f in q:
                avg = 0.5 * (f.select(2 - d, 0) + f.select(2 - d, n))
                f.select(2 - d, 0).copy_(avg)
                f.select(2 - d, n).copy_(avg)
            for t in (0, n):
                for f, v in zip(pr, self.primitives([self.cut(x, d, t, t + 1) for x in q])):
                    self.cut(f, d, t, t + 1).copy_(v)
            halos[d] = (lo + self.primitives(lo), hi + self.primitives(hi))
        return halos

    def split(self, d, q, pr):
        th, dxi, jb, eps = self.th, self.rd[d], self.jac, 0.04
        r, u, p, T = pr[0], pr[1:4], pr[4], pr[5]
        uu = dxi * u[d]
        gm2 = 0.5 / GAMMA
        css = torch.sqrt(T) / th.mach
        csa = css * dxi
        lm = [uu, uu + csa, uu - csa]
        lp = [0.5 * (x + torch.sqrt(x * x + eps * eps)) for x in lm]
        fhi = 0.5 * (GAMMA - 1) * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        full = [jb * (q[m] * uu + (dxi * p if m == d + 1 else 0.0)) for m in range(4)] + [jb * (q[4] + p) * uu]
        ratio = uu / csa
        out = []
        for side, l in ((0, lp), (1, [x - y for x, y in zip(lm, lp)])):
            v1, v2, v3 = l[0], l[1] - l[2], 2.0 * l[0] - l[1] - l[2]
            v4 = v1 - v3 * gm2
            f = [jb * r * v4]
            for c in range(3):
                f.append(jb * r * (v4 * u[c] + (v2 * css * gm2 if c == d else 0.0)))
            f.append(jb * (v1 * q[4] + r * (v2 * uu / dxi * css * gm2 - v3 * (fhi + css * css) * gm2 / (GAMMA - 1))))
            whole, none = (ratio >= 1, ratio <= -1) if side == 0 else (ratio <= -1, ratio >= 1)
            out.append([torch.where(whole, a, torch.where(none, torch.zeros_like(b), b)) for a, b in zip(full, f)])
        return out

    def shocks(self, dv, p):
        div = dv[0][0] + dv[1][1] + dv[2][2]
        vort = (dv[2][1] - dv[1][2]) ** 2 + (dv[0][2] - dv[2][0]) ** 2 + (dv[1][0] - dv[0][1]) ** 2
        dmax = None
        for d in range(3):
            e = self.pext[d]
            pp, pm = self.cut(e, d, HM + 1, HM + 2 + self.n[d]), self.cut(e, d, HM - 1, HM + self.n[d])
            dd = (pp - 2 * p + pm).abs() / (pp + 2 * p + pm)
            dmax = dd if dmax is None else torch.maximum(dmax, dd)
        ssf = div ** 2 / (div ** 2 + vort + 1.0e-30) * dmax
        mx = ssf
        for d in range(3):
            e = self.wrap(ssf, d)
            for off in range(-HM + 1, HM + 1):
                mx = torch.maximum(mx, self.cut(e, d, HM + off, HM + off + self.n[d] + 1))
        return mx > self.case["shkcrt"]

    def roe(self, d, a, b):
        """Left and right eigenvectors of the interfaces between nodes a and b ((rho, u, p, E) each)."""
        w = torch.sqrt(a[0]) / (torch.sqrt(a[0]) + torch.sqrt(b[0]))
        u = [w * a[1 + c] + (1 - w) * b[1 + c] for c in range(3)]
        k = 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        h = w * (a[5] + a[4]) / a[0] + (1 - w) * (b[5] + b[4]) / b[0]
        c = torch.sqrt((GAMMA - 1) * (h - k))
        b1 = (GAMMA - 1) / (c * c)
        b2 = 1 + 2 * b1 * k - b1 * h
        z, one = torch.zeros_like(c), torch.ones_like(c)
        e = [one if i == d else z for i in range(3)]
        L = [[0.5 * (b2 + u[d] / c)] + [-0.5 * (b1 * u[i] + e[i] / c) for i in range(3)] + [0.5 * b1],
             [1 - b2] + [b1 * u[i] for i in range(3)] + [-b1]]
        R = [[one] + [u[i] - c * e[i] for i in range(3)] + [h - u[d] * c], [one] + u + [h - 1 / b1]]
        for i in range(3):                           # shear waves of the two tangential momenta
            if i != d:
                L.append([-u[i]] + [one if m == i else z for m in range(3)] + [z])
                R.append([z] + [one if m == i else z for m in range(3)] + [u[i]])
        L.append([0.5 * (b2 - u[d] / c)] + [-0.5 * (b1 * u[i] - e[i] / c) for i in range(3)] + [0.5 * b1])
        R.append([one] + [u[i] + c * e[i] for i in range(3)] + [h + u[d] * c])
        return L, R

    def upwind(self, d, q, pr, lsh):
        """Interface fluxes -1..N along d from the line-extended q and primitives."""
        n, ax = self.n[d], 2 - d
        fp, fm = self.split(d, q, pr)
        hp = [_along(self.W[d][0], f, d) for f in fp]
        hm = [_along(self.W[d][1], f, d) for f in fm]
        i = torch.arange(-1, n + 1, device="cuda")
        st = lambda f, off: f.index_select(ax, i + off + HM)  # noqa: E731
        up = [[st(f, k - 2) for k in range(5)] for f in fp]
        um = [[st(f, 3 - k) for k in range(5)] for f in fm]
        if not self.case["char"]:
            yes = torch.ones_like(hp[0], dtype=torch.bool)
            return [_mp5(up[m], hp[m], yes) + _mp5(um[m], hm[m], yes) for m in range(5)]
        shock = lsh.index_select(ax, i.clamp(min=0)) | lsh.index_select(ax, (i + 1).clamp(max=n))
        node = lambda off: [st(x, off) for x in (*pr[:5], q[4])]  # noqa: E731
        L, R = self.roe(d, node(0), node(1))
        dot = lambda row, v: sum(r * x for r, x in zip(row, v))  # noqa: E731
        fc = []
        for m in range(5):
            pl = [dot(L[m], [up[c][k] for c in range(5)]) for k in range(5)]
            mi = [dot(L[m], [um[c][k] for c in range(5)]) for k in range(5)]
            fc.append(_mp5(pl, dot(L[m], hp), shock) + _mp5(mi, dot(L[m], hm), shock))
        return [dot([R[m][c] for m in range(5)], fc) for c in range(5)]

    def rhs(self, q, pr, halos):
        n, jb = self.n, self.jac

        def ext(f, d, which):
            if d not in halos:
                return self.wrap(f, d)
            return torch.cat([halos[d][0][which], f, halos[d][1][which]], 2 - d)

        u, p, T = pr[1:4], pr[4], pr[5]
        G = [[_along(self.D[d], ext(u[a], d, 6 + a), d) * self.rd[d] for d in range(3)] for a in range(3)]
        GT = [_along(self.D[d], ext(T, d, 10), d) * self.rd[d] for d in range(3)]
        R = [torch.zeros_like(p) for _ in range(5)]
        lsh = None
        if self.case["char"]:
            self.pext = [ext(p, d, 9) for d in range(3)]
            lsh = self.shocks(G, p)
        for d in range(3):
            qe = [ext(q[m], d, m) for m in range(5)]
            pe = [ext(pr[m], d, 5 + m) for m in range(6)]
            if self.case["conschm"] == 543:
                fh = self.upwind(d, qe, pe, lsh)
                for m in range(5):
                    R[m] -= self.cut(fh[m], d, 1, n[d] + 2) - self.cut(fh[m], d, 0, n[d] + 1)
                continue
            uu = self.rd[d] * pe[1 + d]
            for m in range(5):
                f = jb * (qe[m] * uu + (self.rd[d] * pe[4] if m == d + 1 else pe[4] * uu if m == 4 else 0.0))
                R[m] -= _along(self.D[d], f, d)
        sig, qf = self.th.viscous(G, GT, u, T)
        for d in range(3):
            for m in range(4):
                f = (sig[d][m] if m < 3 else qf[d]) * (self.rd[d] * jb)
                R[1 + m] += _along(self.D[d], self.wrap(f, d), d)
        return R

    def run(self, q, dt, nsteps):
        q = [x.clone() for x in q]
        pr = self.primitives(q)
        for _ in range(nsteps):
            for s, (c1, c2, c3) in enumerate(RK):
                for d in range(3):
                    q = [_along(self.F[d], x, d) for x in q]
                self.walls(q, pr)
                halos = self.swap(q, pr)
                R = self.rhs(q, pr, halos)
                if s == 0:
                    start = [x.clone() for x in q]
                q = [c1 * start[m] + c2 * q[m] + c3 * dt * R[m] / self.jac for m in range(5)]
                pr = self.primitives(q)
        return q


def exact(case, seed):
    torch.backends.cuda.matmul.allow_tf32 = False
    kind = case["kind"]
    if kind == "ensemble":
        res = []
        for b, m in enumerate(_ints(case["boxes"])):
            n = (m,) * 3
            q, box = _flow(n, seed * 64 + b, case["mach"]), _BoxStep(n, case)
            for _ in range(case["nsteps"]):
                q = box.step(q, _dt(n, case["mach"]))
            res.append(list(q))
        return res
    n = _dims(case)
    if kind == "lines":
        nt, f, res = _ints(case["ntype"]), _field(n, case["nf"], seed), []
        for d in range(3):
            g = f
            for a in range(3):
                if a != d:
                    g = g.narrow(3 - a, HM, n[a] + 1)
            scale = n[d] / (2 * math.pi)
            if case["op"] == "central":
                mats = [_deriv_matrix(n[d], nt[d]) * scale]
            elif case["op"] == "filter":
                mats = [_filter_matrix(n[d], nt[d], 0.98)]
            else:
                mats = [_flux_matrix(n[d], nt[d], w, 0.3) for w in "+-"]
                if case["op"] == "fluxdiff":
                    mats = [(M[1:] - M[:-1]) * scale for M in mats]
            for M in mats:
                res.append(_fortran(torch.stack([_along(_cuda(M), x, d) for x in g])))
        return res
    walls = tuple(t != 3 for t in _ints(case.get("ntype", "3,3,3")))
    q, dt = _flow(n, seed, case["mach"], walls), _dt(n, case["mach"])
    if kind == "full":
        return _FullStep(n, case).run(q, dt, case["nsteps"])
    box = _BoxStep(n, case)
    if kind == "adjoint":
        q = q.requires_grad_(True)
        x = q
        for _ in range(case["nsteps"]):
            x = box.step(x, dt)
        J = sum((0.5 * x[1 + c] ** 2 / x[0])[1:, 1:, 1:].sum() for c in range(3)) / math.prod(n)
        J.backward()
        g = _fortran(q.grad)
        return [J.detach()] + [g[..., m] for m in range(5)]
    for _ in range(case["nsteps"]):
        last, q = q, box.step(q, dt)
    if kind == "host":
        return [_fortran(x).cpu().numpy() for x in q] + [box.diagnostics(last)]
    return list(q)
