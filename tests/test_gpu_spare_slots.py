"""Engines with more slots than solves, as a server's is: the solves' clusters
find their slots wherever they are, and empty slots cost no launches' time."""
import time

import numpy as np
import pytest

import oracle
import parfiles
import pkg


@pytest.mark.gpu
@pytest.mark.parametrize("keep", [[39], [0, 17, 38], list(range(1, 40, 2))])
def test_sparse_slots(keep, tmp_par_dir):
    """40 slots filled, some of them kept: in the last slot, a few far apart, a
    number between two launch sizes; then the others filled again."""
    m = pkg.load()

    def problem(k):
        n, radius = 24 + 2 * (k % 5), 1 + k % 3
        return parfiles.orszag_tang(n, radius) if k % 2 else parfiles.blast(n, radius, p_ratio=50.0 + 10 * k, theta=0.1 * k)
    pars = [parfiles.make(tmp_par_dir, f"sparse{k}", problem(k)) for k in range(40)]
    b = m.Batch(40, 40 * max(m.Batch.tiles_for(m.par_load(p)[0]) for p in pars), fp_mode=m.FP_STRICT)
    held = {}

    def add(p):
        k = b.add_par(p)
        b.set_time(k, 0.0, 1e30)
        held[k] = oracle.Oracle(p)

    def step():
        b.run(max_steps=1)
        for k, o in held.items():
            o.advance(o.cfl())
            U, V, S = b.download(k)
            np.testing.assert_array_equal(U, o.U())
            np.testing.assert_array_equal(V, o.V())
            np.testing.assert_array_equal(S, o.scheme())
    for p in pars:
        add(p)
    for k in set(held) - set(keep):
        b.remove(k)
        held.pop(k).close()
    step()
    step()
    for p in pars[:40 - len(keep)]:
        add(p)
    step()
    for o in held.values():
        o.close()
    b.close()


def _per_step(m, par, tiles, slots):
    b = m.Batch(slots, tiles)
    k = b.add_par(par)
    times = []
    for _ in range(5):
        b.set_time(k, 0.0, 1e30)
        t = time.perf_counter()
        b.run(max_steps=20)
        times.append(time.perf_counter() - t)
    b.close()
    return min(times[1:])


@pytest.mark.gpu
def test_spare_slots_cost_little(tmp_par_dir):
    """A step of one small blast among 4,000 slots against one among 20: 1.09
    times as long (1.82 with a cluster for every slot)."""
    m = pkg.load()
    par = parfiles.make(tmp_par_dir, "spare", parfiles.blast(64, 2, p_ratio=100.0))
    tiles = m.Batch.tiles_for(m.par_load(par)[0])
    assert _per_step(m, par, tiles, 4000) < 1.4 * _per_step(m, par, tiles, 20)


@pytest.mark.gpu
def test_a_lone_solve_has_the_cluster_of_its_own_handle(tmp_par_dir):
    """A step of one small blast among 20 slots takes as long as one of a single
    slot (1.32 times with clusters of eight blocks instead of sixteen)."""
    m = pkg.load()
    par = parfiles.make(tmp_par_dir, "lone", parfiles.blast(64, 2, p_ratio=100.0))
    tiles = m.Batch.tiles_for(m.par_load(par)[0])
    assert _per_step(m, par, tiles, 20) < 1.16 * _per_step(m, par, tiles, 1)
