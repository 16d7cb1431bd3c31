"""Setting the clock takes no step: the uploaded ghosts come back until a step
runs, and a clock set back after an upload does not hide the steps taken since."""
import numpy as np
import pytest

from gaukuk_b200 import problems
from gaukuk_b200.config import Params

pytestmark = pytest.mark.gpu


SHAPES = {"run1d": (37, 1, False), "row": (1031, 1, False), "fused2d": (19, 23, False), "five": (18, 27, True)}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_a_clock_that_is_set_takes_no_step(name):
    from gaukuk_b200.sim import Sim
    nx, ny, vz = SHAPES[name]
    p = Params(nx=nx, ny=ny, bc=(1, 1, 2, 3, 1, 1), integrator=2, tmax=1.0, dtoutput=1.0)
    c = problems.random_smooth(p, seed=nx + ny, with_vz=vz)
    g = p.ng
    rng = np.random.default_rng(3)
    for n in (0, 1, 2, 4):
        c[n, g, :, :g] = rng.uniform(1, 2, (p.leny, g))
        c[n, g, :, g + p.nx:] = rng.uniform(1, 2, (p.leny, g))
    with Sim(p, c, mode="parity") as s:
        s.set_time(0.25, 100)
        assert np.array_equal(s.download()[:, g], c[:, g])
        s.run_steps(3)
        want = s.download()
        assert s.get_step() == 103
        s.upload(c)
        s.set_time(0.0, 0)
        s.run_steps(3)
        assert np.array_equal(s.download(), want)
