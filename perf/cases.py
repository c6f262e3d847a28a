"""The time-step path as its users run it: what is timed, on which inputs.

Kinds of case (``case["kind"]``):

* ``solve``   -- a solve set up on the device and advanced by the library's own
  time loop (``Solver.upload_ic``, ``set_time``, ``step``): the reference's
  ``mhd_driver`` with the state resident on the GPU.
* ``driver``  -- the same solve with the time loop kept by the caller: one
  ``cfl_computedt`` and one ``timeStep_advanceSolution`` per step, as the
  Fortran driver calls them.
* ``host``    -- the drop-in on host arrays: ``cfl_computedt`` and
  ``advance_host`` on a pinned U that travels both ways every step.
* ``batch``   -- independent solves of uneven sizes advanced together
  (``hosono_batch_*``), initial states built on the device.
* ``serve``   -- a burst of requests of mixed problems, sizes and radii through
  the request server, from submission to the last result.
* ``riemann`` -- the HLLC module alone on a list of faces in device memory.

Problems are the three the package's configurations hold (Orszag-Tang, Sedov,
MHD blast); the seed moves their free parameters within the ranges of the
committed manifests, so another seed is another flow on the same grid.
"""
import ctypes
import importlib
import math
import os
import random
import tempfile

import numpy as np
import torch

pkg = importlib.import_module("hosono-2dmhd_b200")
problems = importlib.import_module("hosono-2dmhd_b200.problems")
serve = importlib.import_module("hosono-2dmhd_b200.serve")

DOWNLOAD_CELLS = 256 * 256  # a solve up to this size hands its arrays to the host, a larger one stays on the device


def listed():
    return [
        # the smallest calls: a Fortran driver stepping a small blast, two library calls per step
        dict(name="driver_blast64_r2", kind="driver", problem="blast", nx=64, ny=64, radius=2, ell=6.0, steps=8),
        # the reference's own runnable case, from its initial state to t_end = 0.5 (about 200 steps)
        dict(name="ot128_r1_to_end", kind="solve", problem="ot", nx=128, ny=128, radius=1, ell=6.0, steps=0),
        # an ordinary shock problem at the highest order, 7th -> 1st
        dict(name="blast256_r3", kind="solve", problem="blast", nx=256, ny=256, radius=3, ell=6.0, steps=20),
        # odd sizes that are no multiple of any tile, hydrodynamics, outflow boundaries
        dict(name="sedov481x337_r2", kind="solve", problem="sedov", nx=481, ny=337, radius=2, ell=6.0, steps=20),
        # the arithmetic with FMA contraction, on an uneven smooth grid
        dict(name="ot1000x600_r2_fast", kind="solve", problem="ot", nx=1000, ny=600, radius=2, ell=6.0, steps=6,
             fast=True),
        # a large strong-shock hydro run
        dict(name="sedov1024_r2", kind="solve", problem="sedov", nx=1024, ny=1024, radius=2, ell=6.0, steps=8),
        # the benchmark workload, the largest: Orszag-Tang 2048^2 with ell/dx = 12
        dict(name="ot2048_r2", kind="solve", problem="ot", nx=2048, ny=2048, radius=2, ell=12.0, steps=3),
        # the drop-in of a program that keeps its state on the host
        dict(name="host_ot1024_r2", kind="host", problem="ot", nx=1024, ny=1024, radius=2, ell=12.0, steps=1),
        # a parameter study: uneven MHD blasts in one batch
        dict(name="batch_blast16_r2", kind="batch", problem="blast", count=16, nmin=96, nmax=320, radius=2, ell=6.0,
             steps=30),
        # a burst of ten mixed requests on a running server
        dict(name="serve_mixed10", kind="serve", count=10, nmin=64, nmax=256, radius=0, ell=6.0, steps=40),
        # the Riemann solver module on a list of a million faces
        dict(name="riemann_1m", kind="riemann", n=1 << 20, hydro=False, dir=0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "driver", "host", "batch", "serve", "riemann"])
    if kind == "riemann":
        return dict(kind=kind, n=log_int(1000, 1 << 20), hydro=rng.random() < 0.3, dir=rng.randrange(2))
    radius = rng.choice([1, 2, 2, 3])
    ell = rng.choice([6.0, 6.0, 12.0]) if radius == 2 else 6.0
    if kind == "batch":
        nmin = log_int(48, 128)
        return dict(kind=kind, problem=rng.choice(["blast", "ot", "sedov"]), count=rng.randint(2, 16), nmin=nmin,
                    nmax=nmin + rng.randint(16, 200), radius=radius, ell=ell, steps=rng.randint(5, 30))
    if kind == "serve":
        nmin = log_int(48, 96)
        return dict(kind=kind, count=rng.randint(2, 12), nmin=nmin, nmax=nmin + rng.randint(16, 160), radius=0, ell=6.0,
                    steps=rng.randint(5, 40))
    if kind == "host":
        return dict(kind=kind, problem="ot", nx=log_int(512, 1400), ny=log_int(512, 1400), radius=2, ell=ell, steps=1)
    nx = log_int(32, 256) if kind == "driver" else log_int(48, 2000)
    ny = max(24, int(nx * rng.uniform(0.6, 1.0)))
    budget = _flops_per_zone(2) * 2048 * 2048 * 3
    steps = max(1, min(rng.randint(4, 20), int(0.9 * budget / (_flops_per_zone(radius) * nx * ny))))
    case = dict(kind=kind, problem=rng.choice(["ot", "sedov", "blast"]), nx=nx, ny=ny, radius=radius, ell=ell, steps=steps)
    if rng.random() < 0.2:
        case["fast"] = True
    return case


# ----------------------------------------------------------------------
def _params(problem, rng):
    """The free parameters of a problem, from the seed."""
    if problem == "ot":
        return dict(u0=rng.uniform(0.9, 1.1), b0=rng.uniform(0.9, 1.1))
    if problem == "sedov":
        return dict(cx=rng.uniform(-0.2, 0.2), cy=rng.uniform(-0.2, 0.2))
    return dict(ratio=math.exp(rng.uniform(math.log(10.0), math.log(1000.0))), theta=rng.uniform(0.0, math.pi / 2))


def _keys(problem, nx, ny, radius, ell, q):
    """.par keys of a problem on an nx x ny grid: the blasts on square cells (the longer side keeps the problem's
    extent), Orszag-Tang on its whole periodic square."""
    n = max(nx, ny)
    if problem == "ot":
        kv = problems.orszag_tang(n, radius, ell=ell)
        kv.update(IC_U0=repr(q["u0"]), IC_B0=repr(q["b0"] / math.sqrt(4 * math.pi)))
    else:
        if problem == "sedov":
            kv = problems.sedov(n, radius, ell=ell)
            kv.update(IC_shockCenter_x=repr(q["cx"]), IC_shockCenter_y=repr(q["cy"]))
        else:
            kv = problems.blast(n, radius, q["ratio"], q["theta"], ell=ell)
        kv.update(grid_xBeg=repr(-0.5 * nx / n), grid_xEnd=repr(0.5 * nx / n), grid_yBeg=repr(-0.5 * ny / n),
                  grid_yEnd=repr(0.5 * ny / n))
    kv.update(grid_Nx=str(nx), grid_Ny=str(ny))
    return kv


def _setup(directory, problem, nx, ny, radius, ell, q, fast):
    """Parameters, GP tables and initial-state description, as a program's start-up makes them."""
    par = problems.make(directory, "case", _keys(problem, nx, ny, radius, ell, q))
    p, run = pkg.par_load(par)
    p.fp_mode = pkg.FP_FAST if fast else pkg.FP_STRICT
    return dict(par=par, p=p, run=run, gp=pkg.par_gp(par, p.max_radius), ic=pkg.ic_describe(par, p))


class _DeviceArray:
    """A view of a solver's memory for torch (n doubles from an address); torch holds this object, and so the
    solver, as long as a tensor on the memory lives."""

    def __init__(self, solver, address, n):
        self.solver = solver
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(address, False), version=3)


def _state_view(solver):
    """U on the device as (8, nyTot, nxTot)."""
    address, pitch, plane = solver.state_layout()
    flat = torch.as_tensor(_DeviceArray(solver, address, 8 * plane), device="cuda")
    return flat.view(8, solver.nyt, pitch)[:, :, :solver.nxt]


def _sizes(case, rng):
    """(problem, n, radius) of the members of a batch or a burst of requests."""
    out = []
    for k in range(case["count"]):
        n = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        if case["kind"] == "serve":
            out.append((("ot", "sedov", "blast")[k % 3], n, 1 + (k // 3) % 2))
        else:
            out.append((case["problem"], n, case["radius"]))
    return out


def _members(case):
    """Sizes belong to the case, not to the seed: every seed costs about the same."""
    return _sizes(case, random.Random(1000 * case["nmin"] + 10 * case["nmax"] + case["count"]))


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "riemann":
        return _prepare_riemann(case, seed)
    fast = bool(case.get("fast"))
    with tempfile.TemporaryDirectory() as d:
        if kind in ("batch", "serve"):
            mem = [_setup(d, prob, n, n, radius, case["ell"], _params(prob, rng), fast)
                   for prob, n, radius in _members(case)]
            if kind == "serve":
                server = serve.Server(memory_budget=2 << 30, max_resident=case["count"])
                return dict(kind=kind, case=case, mem=mem, server=server)
            batch = pkg.Batch(len(mem), sum(pkg.Batch.tiles_for(m["p"]) for m in mem))
            for m in mem:
                m["slot"] = batch.add(m["p"], *m["gp"])
            return dict(kind=kind, case=case, mem=mem, batch=batch)
        s = _setup(d, case["problem"], case["nx"], case["ny"], case["radius"], case["ell"],
                   _params(case["problem"], rng), fast)
        solver = pkg.Solver(s["p"], *s["gp"])
        state = dict(kind=kind, case=case, solver=solver, **s)
        if kind == "host":
            U, V = pkg.ic_set(s["par"], s["p"])
            pinned = torch.empty(U.shape, dtype=torch.float64, pin_memory=True)
            state["U"] = pinned.numpy()
            state["U"][...] = U
            state["pinned"] = pinned
            solver.upload(U, V)
        return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "riemann":
        F = state["F"]
        state["solver"].riemann(state["n"], state["uL"].data_ptr(), state["uR"].data_ptr(), case["dir"], F.data_ptr())
        return F
    if kind == "host":
        dt = state["solver"].cfl_computedt()
        state["solver"].advance_host(dt, state["U"])
        return dict(dt=dt, U=state["U"])
    if kind == "batch":
        b = state["batch"]
        for m in state["mem"]:
            desc, xt, yt = m["ic"]
            b._check(b.lib.hosono_batch_ic(b.h, m["slot"], ctypes.byref(desc), pkg._p(xt), pkg._p(yt)), "ic")
            b.set_time(m["slot"], 0.0, m["run"].tmax)
        b.run(case["steps"])
        return [(b.status(m["slot"])["t"],) + b.download(m["slot"]) for m in state["mem"]]
    if kind == "serve":
        s = state["server"]
        ids = [s.submit_ic(m["p"], *m["gp"], *m["ic"], m["run"].tmax, nstepmax=case["steps"]) for m in state["mem"]]
        done = [s.wait(i) for i in ids]
        return [(info["t"], info["nstep"], U) for info, U, _, _ in done]
    solver = state["solver"]
    solver.upload_ic(*state["ic"])
    if kind == "driver":
        t = 0.0
        for _ in range(case["steps"]):
            dt = solver.cfl_computedt()
            solver.timeStep_advanceSolution(dt)
            t += dt
        n = case["steps"]
    else:
        solver.set_time(0.0, state["run"].tmax)
        t, n = solver.step(case["steps"] if case["steps"] > 0 else 1 << 30)
    if case["nx"] * case["ny"] <= DOWNLOAD_CELLS:
        U, V, scheme = solver.download()
        return dict(t=t, n=n, U=U, V=V, scheme=scheme)
    return dict(t=t, n=n, U=_state_view(solver))


# ----------------------------------------------------------------------
# Riemann faces: left and right states a few tenths apart, one in eight a
# strong jump (up to 1000 : 1 in pressure), as a solve's faces have them.
GAMMA = 5.0 / 3.0


def _faces(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n = case["n"]

    def normal(*shape):
        return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)

    def cons(rho, v, p, b):
        e = p / (GAMMA - 1.0) + 0.5 * rho * (v * v).sum(1) + 0.5 * (b * b).sum(1)
        return torch.cat([rho[:, None], rho[:, None] * v, e[:, None], b], 1).contiguous()

    strong = (torch.rand(n, dtype=torch.float64, device="cuda", generator=g) < 0.125).to(torch.float64)
    size = 0.1 + strong * 1.5
    rho, p, v, b = torch.exp(0.5 * normal(n)), torch.exp(normal(n)), normal(n, 3), normal(n, 3)
    if case["hydro"]:
        b = b * 0.0
    left = cons(rho, v, p, b)
    right = cons(rho * torch.exp(size * normal(n)), v + size[:, None] * normal(n, 3),
                 p * torch.exp(2.0 * size * normal(n)), b + (0.0 if case["hydro"] else 1.0) * 0.1 * normal(n, 3))
    return left, right


def _prepare_riemann(case, seed):
    with tempfile.TemporaryDirectory() as d:
        s = _setup(d, "blast", 24, 24, 1, 6.0, dict(ratio=100.0, theta=0.5), False)
    s["p"].force_hydro = 1 if case["hydro"] else 0
    s["p"].gamma = GAMMA
    left, right = _faces(case, seed)
    return dict(kind="riemann", case=case, solver=pkg.Solver(s["p"], *s["gp"]), n=case["n"], uL=left, uR=right,
                F=torch.empty_like(left))


def _hllc(uL, uR, d, hydro):
    """HLLC for ideal MHD (S. Li, J. Comput. Phys. 203, 2005) with the wave speeds of the left, right and mean state."""
    N, T = 1 + d, 2 - d
    bN, bT = 5 + d, 6 - d

    def prim(U):
        v = U[1:4] / U[0]
        b = U[5:8] * (0.0 if hydro else 1.0)
        p = np.maximum((GAMMA - 1.0) * (U[4] - 0.5 * (b * b).sum(0) - 0.5 * U[0] * (v * v).sum(0)), 1e-12)
        return U[0], v, p, b

    def fast(rho, p, b):
        c = (GAMMA * p + (b * b).sum(0)) / rho
        r = c * c - 4.0 * GAMMA * p * b[d] ** 2 / rho ** 2
        return np.sqrt(np.maximum(1e-14, 0.5 * (c + np.sqrt(np.maximum(r, 0.0)))))

    def flux(U, v, p, b):
        pt = p + 0.5 * (b * b).sum(0)
        F = U * v[d]
        F[1:4] -= b[d] * b
        F[1 + d] += pt
        F[4] += pt * v[d] - b[d] * (v * b).sum(0)
        F[5:8] = 0.0 if hydro else b * v[d] - v * b[d]
        F[5 + d] = 0.0
        return F

    (rL, vL, pL, bL), (rR, vR, pR, bR) = prim(uL), prim(uR)
    vm, cm = 0.5 * (vL[d] + vR[d]), fast(0.5 * (rL + rR), 0.5 * (pL + pR), 0.5 * (bL + bR))
    sL = np.minimum(vL[d] - fast(rL, pL, bL), vm - cm)
    sR = np.maximum(vR[d] + fast(rR, pR, bR), vm + cm)
    ptL, ptR = pL + 0.5 * (bL * bL).sum(0), pR + 0.5 * (bR * bR).sum(0)
    dL, dR = sL - vL[d], sR - vR[d]
    s = (uR[N] * dR - uL[N] * dL + ptL - ptR - bL[d] ** 2 + bR[d] ** 2) / (rR * dR - rL * dL)
    fL, fR = flux(uL, vL, pL, bL), flux(uR, vR, pR, bR)
    h = (sR * uR - sL * uL + fL - fR) / (sR - sL)
    bh = np.zeros_like(bL) if hydro else h[5:8]
    vbh = (bh * (h[1:4] / h[0])).sum(0)
    pst = rL * dL * (s - vL[d]) + ptL - bL[d] ** 2 + bh[d] ** 2

    def star(U, r, v, b, pt, sK, dK):
        w = sK - s
        W = np.empty_like(U)
        W[0] = r * dK / w
        W[N] = W[0] * s
        W[T] = W[0] * v[1 - d] - (bh[d] * bh[1 - d] - b[d] * b[1 - d]) / w
        W[3] = W[0] * v[2] - (bh[d] * bh[2] - b[d] * b[2]) / w
        W[4] = (U[4] * dK + pst * s - pt * v[d] - bh[d] * vbh + b[d] * (b * v).sum(0)) / w
        W[bN], W[bT], W[7] = bh[d], bh[1 - d], bh[2]
        return W

    left = fL + sL * (star(uL, rL, vL, bL, ptL, sL, dL) - uL)
    right = fR + sR * (star(uR, rR, vR, bR, ptR, sR, dR) - uR)
    return np.where(sL > 0.0, fL, np.where(s > 0.0, left, np.where(sR >= 0.0, right, fR)))


def exact(case, seed):
    """The module's values in plain 64-bit numpy.  The whole-step cases have
    none here: a GP-MOOD step in numpy, quad-precision GP tables included,
    takes minutes at these sizes (the repository's tests hold it bit for bit
    against the C++ oracle instead)."""
    if case["kind"] != "riemann":
        return None
    left, right = _faces(case, seed)
    F = _hllc(left.cpu().numpy().T.copy(), right.cpu().numpy().T.copy(), case["dir"], case["hydro"])
    return np.ascontiguousarray(F.T)


# ----------------------------------------------------------------------
def _flops_per_zone(radius):
    """FP64 operations per interior cell and time step without any lowered
    cell: three stages of 8-variable GP sums on 1 + 2R(R+1) points for
    R + 1 quadrature points of four face sides, 2 (R + 1) Riemann solves of
    about 465 operations, and the update and detection; then the RK combines
    and the CFL reduction."""
    ns, nq = 1 + 2 * radius * (radius + 1), radius + 1
    return 3 * (64 * ns * nq + 930 * nq + 226) + 92


def work(case):
    """State in and out once per pass; the operations of its steps."""
    if case["kind"] == "riemann":
        return dict(bytes=24.0 * 8 * case["n"], flops=465.0 * case["n"])
    if case["kind"] in ("batch", "serve"):
        cells = [(n * n, radius) for _, n, radius in _members(case)]
        return dict(bytes=float(sum(16 * 8 * c for c, _ in cells)),
                    flops=float(sum(c * case["steps"] * _flops_per_zone(r) for c, r in cells)))
    c = case["nx"] * case["ny"]
    steps = case["steps"] if case["steps"] > 0 else 208
    return dict(bytes=16.0 * 8 * c, flops=float(c) * steps * _flops_per_zone(case["radius"]))
