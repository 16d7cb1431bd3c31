"""A second upload on a handle that has run: a z momentum that appears or goes must
not leave the captured steps of the first state in use, nor what they left in the
stage buffers in a frame.  70 steps are whole graphs and a remainder; state and dt
sequence are those of a fresh handle."""
import numpy as np
import pytest

from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,integrator,path", [
    (64, 1, 1, "run1d"), (64, 1, 2, "run1d"), (600, 1, 3, "run1d"), (1100, 1, 1, "generic"),
    (1100, 1, 2, "generic"), (1100, 1, 3, "generic"), (40, 24, 1, "generic"), (40, 24, 2, None)])
@pytest.mark.parametrize("first_vz", [False, True])
def test_second_upload_is_a_fresh_handle(nx, ny, integrator, path, first_vz):
    from gaukuk_b200.sim import Sim
    p = Params(nx=nx, ny=ny, bc=(1, 1, 2, 3, 1, 1), integrator=integrator, tmax=100.0, dtoutput=100.0)
    first = problems.random_smooth(p, seed=1, with_vz=first_vz)
    second = problems.random_smooth(p, seed=2, with_vz=not first_vz)
    second[3] *= 8.0  # z momentum sets the CFL speed
    second[4] *= 40.0
    with Sim(p, first, mode="parity") as s:
        assert path is None or s.path == path
        s.run_steps(70)
        s.upload(second)
        assert path is None or s.path == path
        s.run_steps(70)
        got, dts = active(p, s.download()).copy(), s.dt_log()
    with Sim(p, second, mode="parity") as s:
        s.run_steps(70)
        assert dts == s.dt_log() and len(dts) == 70
        assert np.array_equal(got, active(p, s.download()))


@pytest.mark.parametrize("nx,ny,bc", [(1, 1, (1, 1)), (1, 1, (2, 3)), (40, 24, (1, 1)), (40, 24, (2, 3))])
@pytest.mark.parametrize("integrator", [2, 3])
def test_second_upload_leaves_no_trace_in_a_frame(nx, ny, bc, integrator):
    from gaukuk_b200.sim import Sim
    p = Params(nx=nx, ny=ny, bc=bc + (1, 1, 1, 1), integrator=integrator, tmax=100.0, dtoutput=100.0)
    second = problems.random_smooth(p, seed=2)
    with Sim(p, problems.random_smooth(p, seed=1, with_vz=True), mode="parity") as s:
        s.run_steps(3)
        s.upload(second)
        s.run_steps(1)
        got = s.download()
    with Sim(p, second, mode="parity") as s:
        s.run_steps(1)
        assert np.array_equal(got, s.download())
