"""A call that returns with an error has none of its work left on the stream:
the caller's buffers and the state are the caller's again."""
import pytest

import parfiles
import pkg


@pytest.mark.gpu
@pytest.mark.parametrize("bands", [1, 8])
def test_failed_advance_host_leaves_an_idle_stream(bands, tmp_par_dir):
    """A step stopped by its pass cap rebuilds V from the uploaded U before it returns."""
    import torch

    m = pkg.load()
    par = parfiles.make(tmp_par_dir, f"idle{bands}", parfiles.blast(2048, 1, p_ratio=1000.0))
    s = m.Solver.from_par(par)
    s.set_tuning(upload_bands=bands)
    U = torch.empty(s.download()[0].shape, dtype=torch.float64, pin_memory=True).numpy()
    U[...] = s.download()[0]
    dt = s.cfl_computedt()
    s.set_mood_cap(1)
    for _ in range(3):
        stream = torch.cuda.ExternalStream(s.stream())
        with pytest.raises(m.HosonoError) as e:
            s.advance_host(dt, U)
        idle = stream.query()
        assert e.value.code == m.EMOODCAP
        assert idle
    s.set_mood_cap(0)
    s.advance_host(dt, U)
    s.close()
