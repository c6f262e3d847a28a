"""The kernels a step graph is said to have launched are those that the same
steps launch one by one from the host, where each is counted."""
import pytest

import parfiles
import pkg

RUNS = {
    "chain": lambda: parfiles.blast(512, 3, p_ratio=1000.0, theta=0.4),
    "chain_r1": lambda: parfiles.blast(640, 1, p_ratio=1000.0, theta=1.1),
    "clusters": lambda: parfiles.blast(64, 3, p_ratio=100.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("later", [0, 1])
@pytest.mark.parametrize("case", sorted(RUNS))
def test_graph_counts_equal_host_counts(case, later, tmp_par_dir):
    m = pkg.load()
    par = parfiles.make(tmp_par_dir, f"count_{case}{later}", RUNS[case]())
    counts = []
    for graphs in (True, False):
        s = m.Solver.from_par(par)
        s.set_graphs(graphs)
        s.set_tuning(later_passes=later)
        s.set_time(0.0, 1e30)
        s.step(60)  # the blast's front grows past the clusters' share
        got = []
        for _ in range(4):
            dt = s.cfl_computedt()
            s.profile_read(reset=True)
            s.timeStep_advanceSolution(dt)
            got.append(s.profile_read(reset=True)[2])
        s.set_time(0.0, 1e30)
        s.step(1)
        got.append(s.profile_read(reset=True)[2])
        counts.append(got)
        s.close()
    assert counts[0] == counts[1]
    assert later or (max(counts[0]) > 30) == (case != "clusters")


@pytest.mark.gpu
def test_banded_upload_counts_its_kernels(tmp_par_dir):
    """Eight bands: a conversion and a pass 1 each, instead of one of either."""
    m = pkg.load()
    par = parfiles.make(tmp_par_dir, "count_bands", parfiles.orszag_tang(128, 2))
    counts = []
    for bands in (1, 8):
        s = m.Solver.from_par(par)
        s.set_tuning(upload_bands=bands)
        U = s.download()[0]
        dt = s.cfl_computedt()
        s.profile_read(reset=True)
        s.advance_host(dt, U)
        counts.append(s.profile_read(reset=True)[2])
        s.close()
    assert counts[1] - counts[0] == 8 * 2 - 2
