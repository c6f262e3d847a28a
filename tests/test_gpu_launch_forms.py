"""Pass 1's launch geometry under each launch choice."""
import pytest

import parfiles
import pkg


def _solver(tmp_par_dir, n, radius):
    m = pkg.load()
    return m.Solver.from_par(parfiles.make(tmp_par_dir, f"form{n}_{radius}", parfiles.orszag_tang(n, radius)))


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [1, 2, 3])
def test_reported_grid_is_the_launched_one(radius, tmp_par_dir):
    """A new handle's pass 1: two blocks an SM over many tiles, quarter tiles
    where there are few."""
    s = _solver(tmp_par_dir, 512, radius)
    info = s.launch_info()
    assert info["pass1_grid"] == 2 * info["sms"]
    s.close()
    s = _solver(tmp_par_dir, 24, radius)
    info = s.launch_info()
    assert info["pass1_grid"] == 4 * info["tiles"] < 2 * info["sms"]
    s.close()
