"""The forms a step's kernels take by size and data, each bit for bit against
the oracle (strict arithmetic; equality, so no tolerance): MOOD passes in one
cluster per instance and in the kernel chain, alone and side by side in a
batch; pass 1 on whole, half and quarter tiles; its solver modes by what a
tile's planes hold; the Riemann module at the edges of the shared-denominator
range and on unaligned arrays; a run whose steps turn over on the device."""
import numpy as np
import pytest

import oracle
import parfiles
import pkg


def _same(s, o):
    U, V, S = s.download()
    np.testing.assert_array_equal(U, o.U())
    np.testing.assert_array_equal(V, o.V())
    np.testing.assert_array_equal(S, o.scheme())


# 24: every stencil reaches a boundary, 3 tiles in quarters; 200: below two
# tiles per block; 330: whole tiles.  The blasts lower some 2 cells per cell of
# their front and pass: 330^2 is above the cluster's share, the others below.
RUNS = {
    "ot24_r1": (lambda: parfiles.orszag_tang(24, 1), 4),
    "sedov24_r3": (lambda: parfiles.sedov(24, 3), 6),
    "blast200_r1": (lambda: parfiles.blast(200, 1, p_ratio=1000.0, theta=0.4), 4),
    "blast330_r2": (lambda: parfiles.blast(330, 2, p_ratio=1000.0, theta=0.7), 6),
    "blast300_r3": (lambda: parfiles.blast(300, 3, p_ratio=800.0, theta=0.2), 4),
}


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(RUNS))
def test_run_matches_stepwise_oracle(case, tmp_par_dir):
    """All steps in one launch (the next step begins inside it), then one step
    with the caller's dt."""
    m = pkg.load()
    kv, steps = RUNS[case]
    par = parfiles.make(tmp_par_dir, "forms_" + case, kv())
    o = oracle.Oracle(par)
    s = m.Solver.from_par(par, fp_mode=m.FP_STRICT)
    s.set_time(0.0, 1e30)
    for _ in range(steps):
        o.advance(o.cfl())
    t, n = s.step(steps)
    assert n == steps
    _same(s, o)
    dt = s.cfl_computedt()
    assert dt == o.cfl()
    o.advance(dt)
    s.timeStep_advanceSolution(dt)
    _same(s, o)
    s.close()
    o.close()


@pytest.mark.gpu
def test_cluster_and_chain_share_a_batch(tmp_par_dir):
    """One instance with long work lists beside small ones of other radii and
    boundaries: the chain takes the first in the stages where the clusters take
    the rest."""
    m = pkg.load()
    kvs = [parfiles.blast(330, 2, p_ratio=1000.0, theta=0.7), parfiles.blast(48, 2, p_ratio=300.0, theta=0.2),
           parfiles.orszag_tang(40, 1), parfiles.sedov(36, 3), parfiles.blast(64, 1, p_ratio=50.0, theta=1.2)]
    pars = [parfiles.make(tmp_par_dir, f"mix{i}", kv) for i, kv in enumerate(kvs)]
    b = m.Batch(len(pars) + 7, sum(m.Batch.tiles_for(m.par_load(p)[0]) for p in pars) + 11, fp_mode=m.FP_STRICT)
    slots = [b.add_par(p) for p in pars]
    for k in slots:
        b.set_time(k, 0.0, 1e30)
    b.run(max_steps=4)
    for k, p in zip(slots, pars):
        o = oracle.Oracle(p)
        for _ in range(4):
            o.advance(o.cfl())
        U, V, S = b.download(k)
        np.testing.assert_array_equal(U, o.U())
        np.testing.assert_array_equal(V, o.V())
        np.testing.assert_array_equal(S, o.scheme())
        o.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("first", [0, 1, 2])
def test_handed_over_instances_beside_the_chain(first, tmp_par_dir):
    """Blasts whose long passes end at different passes of a stage: the clusters
    take one over, at the front, in the middle and at the back of the batch's
    lists, while the chain still holds the others' recompute list."""
    m = pkg.load()
    kvs = [parfiles.blast(200, 2, p_ratio=1000.0, theta=0.7), parfiles.blast(400, 3, p_ratio=1000.0, theta=0.4),
           parfiles.blast(300, 1, p_ratio=300.0, theta=1.1)]
    kvs = kvs[first:] + kvs[:first] + [parfiles.orszag_tang(40, 1)]
    pars = [parfiles.make(tmp_par_dir, f"hand{i}", kv) for i, kv in enumerate(kvs)]
    b = m.Batch(len(pars), sum(m.Batch.tiles_for(m.par_load(p)[0]) for p in pars), fp_mode=m.FP_STRICT)
    slots = [b.add_par(p) for p in pars]
    for k in slots:
        b.set_time(k, 0.0, 1e30)
    b.run(max_steps=6)
    for k, p in zip(slots, pars):
        o = oracle.Oracle(p)
        for _ in range(6):
            o.advance(o.cfl())
        U, V, S = b.download(k)
        np.testing.assert_array_equal(U, o.U())
        np.testing.assert_array_equal(V, o.V())
        np.testing.assert_array_equal(S, o.scheme())
        o.close()
    b.close()


@pytest.mark.gpu
def test_step_after_autotune(tmp_par_dir):
    """The timing launches leave pass 1's tile counters at their start for a
    step with the caller's dt."""
    m = pkg.load()
    par = parfiles.make(tmp_par_dir, "tuned", parfiles.orszag_tang(96, 2))
    s = m.Solver.from_par(par)
    o = oracle.Oracle(par)
    default = s.tuning()
    s.autotune(trials=1, force=True)
    s.set_tuning(**default)
    dt = o.cfl()
    s.timeStep_advanceSolution(dt)
    o.advance(dt)
    U, V, S = s.download()
    np.testing.assert_array_equal(U, o.U())
    np.testing.assert_array_equal(S, o.scheme())
    s.close()
    o.close()


def _wrap(U, g, periodic):
    """Guard cells from the interior (boundaryConditions_applyBlk)."""
    inner = U[g:-g, g:-g]
    return np.pad(inner, ((g, g), (g, g), (0, 0)), mode="wrap" if periodic else "edge")


# what is added to the problem's planar state: out-of-plane velocity, field
MODES = {
    "mhd_z": ("ot", 0.3, 0.2), "mhd_vz_only": ("ot", 0.3, 0.0), "mhd_bz_half": ("ot", 0.0, 0.2),
    "hydro_vz": ("sedov", 0.3, 0.0), "hydro_field": ("sedov", 0.0, 0.2), "hydro_field_vz": ("sedov", 0.1, 0.2),
}


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [1, 2, 3])
@pytest.mark.parametrize("mode", sorted(MODES))
def test_solver_modes_by_data(mode, radius, tmp_par_dir):
    """States that keep the solver from leaving planes out, on part of the
    grid, so that both kinds of tile meet: out-of-plane velocity or field, and
    a stored field in a hydro run, which its HLL state reads."""
    m = pkg.load()
    prob, vz, bz = MODES[mode]
    kv = parfiles.orszag_tang(72, radius) if prob == "ot" else parfiles.sedov(72, radius)
    par = parfiles.make(tmp_par_dir, f"mode_{mode}_{radius}", kv)
    o = oracle.Oracle(par)
    s = m.Solver.from_par(par, fp_mode=m.FP_STRICT)
    g = s.params.ngc
    U = o.U().copy()
    x = np.arange(U.shape[1])[None, :]
    part = np.where(x < U.shape[1] // 2, np.sin(0.2 * x) ** 2, 0.0) * np.ones((U.shape[0], 1))
    U[..., 3] += vz * part * U[..., 0]
    U[..., 4] += 0.5 * vz * vz * part * part * U[..., 0] + 0.5 * (bz * part) ** 2
    U[..., 7] += bz * part
    U = _wrap(U, g, prob == "ot")
    s.upload(U)
    _, V, _ = s.download()
    o.set_U(U)
    o.set_V(V)
    for _ in range(2):
        dt = o.cfl()
        assert s.cfl_computedt() == dt
        o.advance(dt)
        s.timeStep_advanceSolution(dt)
        _same(s, o)
    s.close()
    o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("hydro,field", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("offset", [0, 1])
def test_riemann_operand_ranges(hydro, field, offset, tmp_par_dir):
    """Face states scaled across the powers of two where the solver leaves the
    shared denominators for IEEE division (densities 2^-100 and 2^101, momenta
    down to 2^-860 and exact zeros), subnormal momenta among them, on arrays
    that start on a 16-byte boundary and eight bytes past one."""
    import torch

    m = pkg.load()
    par = parfiles.make(tmp_par_dir, f"rr{int(hydro)}{int(field)}",
                        parfiles.sedov(8, 1) if hydro else parfiles.orszag_tang(8, 1))
    o = oracle.Oracle(par)
    s = m.Solver.from_par(par, fp_mode=m.FP_STRICT)
    rng = np.random.default_rng(23)
    n = 3000

    def states():
        u = np.zeros((n, 8))
        e = rng.choice([0, 0, 0, -99, -100, -101, 99, 100, 101, 130, -130], size=n).astype(float)
        u[:, 0] = rng.uniform(0.5, 2.0, n) * 2.0 ** e
        v = rng.normal(size=(n, 3)) * rng.choice([1.0, 3.0, 0.0, 2.0 ** -400, 2.0 ** -700, 2.0 ** -861], size=(n, 3))
        u[:, 1:4] = v * u[:, :1]
        u[::97, 2] = 5e-320
        if field:
            u[:, 5:8] = rng.normal(size=(n, 3)) * np.sqrt(u[:, :1]) * rng.choice([1.0, 0.0], size=(n, 3))
        b2 = (u[:, 5:8] ** 2).sum(1) if not hydro else 0.0
        u[:, 4] = 0.5 * (u[:, 1:4] ** 2).sum(1) / u[:, 0] + 0.5 * b2 + rng.uniform(0.1, 3.0, n) * u[:, 0]
        return u
    uL, uR = states(), states()
    uR[: n // 2, 0] = uL[: n // 2, 0] * rng.uniform(0.5, 2.0, n // 2)  # sides of one magnitude
    uR[: n // 2, 4] = 0.5 * (uR[: n // 2, 1:4] ** 2).sum(1) / uR[: n // 2, 0] + uL[: n // 2, 4]

    def dev(a):
        flat = torch.zeros(a.size + 1, dtype=torch.float64, device="cuda")
        flat[offset:offset + a.size] = torch.from_numpy(a.reshape(-1)).cuda()
        return flat
    dL, dR = dev(uL), dev(uR)
    for direction in (0, 1):
        F = torch.zeros(8 * n + 1, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.riemann(n, dL.data_ptr() + 8 * offset, dR.data_ptr() + 8 * offset, direction, F.data_ptr() + 8 * offset)
        got = F.cpu().numpy()[offset:offset + 8 * n].reshape(n, 8)
        ref = np.array([o.hllc(uL[k], uR[k], direction) for k in range(n)])
        np.testing.assert_array_equal(got, ref)
    s.close()
    o.close()
