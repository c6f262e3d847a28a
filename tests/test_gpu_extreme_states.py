"""States at the ends of what 64 bits hold, each bit for bit against the oracle
(strict arithmetic; equality, NaN where it has NaN, so no tolerance)."""
import numpy as np
import pytest

import oracle
import parfiles
import pkg


def _pair(tmp_par_dir, name, kv, edit):
    """The oracle and a solver on the problem's state as `edit` leaves its interior."""
    m = pkg.load()
    par = parfiles.make(tmp_par_dir, name, kv)
    o = oracle.Oracle(par)
    s = m.Solver.from_par(par, fp_mode=m.FP_STRICT)
    g = s.params.ngc
    U = o.U()[g:-g, g:-g].copy()
    edit(U)
    U = np.pad(U, ((g, g), (g, g), (0, 0)), mode="wrap" if "periodic" in kv["sim_BC"] else "edge")
    s.upload(U)
    o.set_U(U)
    o.set_V(s.download()[1])
    return o, s


def _step_alike(o, s, dt, steps=1):
    for _ in range(steps):
        o.advance(dt)
        s.timeStep_advanceSolution(dt)
        U, V, S = s.download()
        np.testing.assert_array_equal(U, o.U())
        np.testing.assert_array_equal(V, o.V())
        np.testing.assert_array_equal(S, o.scheme())


# Two neighbours whose face overflows: the reference's solver then gives NaN in
# variables that its states hold as zeros, a hydro run's field or a planar
# flow's out-of-plane momentum and field.
FACES = {
    "sedov": ([1e200, 1, -2, 0, 1e25, 0, 0, 0], [1e-3, -1e10, -1e10, 0, 1, 0, 0, 0]),
    "ot": ([1e200, 1e10, 1, 0, -1, 0, 1, 0], [2, -1e10, -1e160, 0, 1e300, 1, 1, 0]),
}


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [1, 2, 3])
@pytest.mark.parametrize("prob", sorted(FACES))
def test_overflow_reaches_the_zero_planes(prob, radius, tmp_par_dir):
    def edit(U):
        U[20, 19], U[20, 20] = FACES[prob]
        U[31, 7], U[32, 7] = FACES[prob]
    kv = parfiles.sedov(40, radius) if prob == "sedov" else parfiles.orszag_tang(40, radius)
    o, s = _pair(tmp_par_dir, f"over_{prob}{radius}", kv, edit)
    _step_alike(o, s, 1e-3)
    assert not np.isfinite(o.U()[..., [3, 7] if prob == "ot" else [3, 5, 6, 7]]).all(axis=(0, 1)).any()
    s.close()
    o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("hydro", [True, False])
def test_riemann_non_finite(hydro, tmp_par_dir):
    """The module on faces of extreme, infinite and NaN operands."""
    import torch

    m = pkg.load()
    par = parfiles.make(tmp_par_dir, f"rnf{int(hydro)}",
                        parfiles.sedov(8, 1) if hydro else parfiles.orszag_tang(8, 1))
    o = oracle.Oracle(par)
    s = m.Solver.from_par(par, fp_mode=m.FP_STRICT)
    rng = np.random.default_rng(5)
    n = 6000

    def states():
        u = np.zeros((n, 8))
        u[:, 0] = rng.choice([1.0, 2.0, 1e-3, 1e200, 1e-200, 1e-310, -1.0, 0.0, np.nan, np.inf], n)
        u[:, 1:3] = rng.choice([0.0, 1.0, -2.0, 1e10, -1e10, 1e160, -1e160, 1e300, np.nan, np.inf], (n, 2),
                               p=[.2, .2, .2, .1, .1, .05, .05, .04, .03, .03])
        u[:, 4] = rng.choice([1.0, 0.5e20, 1e25, 1e300, -1.0, np.nan, np.inf], n)
        if not hydro:
            u[:, 5:7] = rng.choice([0.0, 1.0, 1e160, np.nan, np.inf], (n, 2), p=[.4, .4, .1, .05, .05])
        return u
    uL, uR = states(), states()
    for direction in (0, 1):
        dL, dR = torch.from_numpy(uL).cuda(), torch.from_numpy(uR).cuda()
        F = torch.zeros(n, 8, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.riemann(n, dL.data_ptr(), dR.data_ptr(), direction, F.data_ptr())
        ref = np.array([o.hllc(uL[k], uR[k], direction) for k in range(n)])
        np.testing.assert_array_equal(F.cpu().numpy(), ref)
    s.close()
    o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 1e140, 1e153])
def test_pressure_sensor_range(scale, tmp_par_dir):
    """detect's pressure sensor where the products of two pressures leave the
    range of 64 bits (1e153) and where they do not: a noisy converging flow,
    every value of it scaled alike."""
    def edit(U):
        rng = np.random.default_rng(3)
        n = U.shape[0]
        rho, p = rng.uniform(0.8, 1.2, (n, n)), 14.0 * rng.uniform(0.7, 1.3, (n, n))
        x = (np.arange(n) + 0.5) / n - 0.5
        vx, vy = -2.5 * np.sign(x)[None, :] * rng.uniform(0.5, 1.0, (n, n)), -2.5 * np.sin(6 * x)[:, None] + 0 * rho
        U[...] = 0.0
        U[..., 0], U[..., 1], U[..., 2] = rho, rho * vx, rho * vy
        U[..., 4] = p / 0.4 + 0.5 * rho * (vx * vx + vy * vy)
        U *= scale
    o, s = _pair(tmp_par_dir, f"sensor{scale}", parfiles.sedov(40, 2), edit)
    _step_alike(o, s, 1e-3, steps=2)
    assert (o.scheme() < 2).sum() > 100
    s.close()
    o.close()
