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


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [1, 2, 3])
@pytest.mark.parametrize("blocks,boxes", [(2, 1), (2, 2), (3, 1), (4, 1)])
def test_blocks_per_sm_are_resident(blocks, boxes, radius, tmp_par_dir):
    """The blocks an SM that a choice names fit it (three of four at R = 3:
    58 KB each), so its register budget buys the occupancy it is for."""
    s = _solver(tmp_par_dir, 512, radius)
    for staging in (0, 1) if blocks == 2 else (0,):
        s.set_tuning(pass1_staging=staging, pass1_blocks_per_sm=blocks, pass1_boxes=boxes)
        info = s.launch_info()
        assert info["pass1_grid"] == info["sms"] * (3 if radius == 3 and blocks == 4 else blocks)
    s.close()
