"""gk_advance sizes its launches by the last known CFL speed: a step limit inside
the first batch, and speeds that change by much during the call."""
import time

import numpy as np
import pytest

import gk_oracle
from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active

pytestmark = pytest.mark.gpu


def test_a_step_limit_bounds_the_launches():
    """Three steps of a run whose output time is 2^11 steps away.  64 graphs of
    32 steps are 4096 launches, at no less than 0.8 us each 3.3 ms; one graph is
    64 launches and a few steps, well under a third of that."""
    from gaukuk_b200.sim import Sim
    p, c = problems.kh(64, seed=1)
    p = Params(**{**p.__dict__, "stepmax": 3})
    with Sim(p, c, mode="parity") as s:
        dt = p.cfl * (1.0 / 64) / s.cmax()
        s.advance(2048 * dt)  # captures the graph
        best = 1e9
        for _ in range(5):
            s.set_time(0.0, 0)
            t0 = time.perf_counter()
            _, step, cont = s.advance(2048 * dt)
            best = min(best, time.perf_counter() - t0)
            assert (step, cont) == (3, False)
    assert best < 1.1e-3, best


def _pulse(nx, ny, hot):
    """A hot spot in a cold gas (its speed falls), or a converging flow (its
    speed rises)."""
    p = Params(nx=nx, ny=ny, bc=(2, 2, 2, 2, 1, 1), integrator=2, tmax=1.0, dtoutput=1.0)
    x = (np.arange(nx) + 0.5)[None, None, :] / nx * np.ones((1, ny, nx))
    y = (np.arange(ny) + 0.5)[None, :, None] / ny * np.ones((1, ny, nx))
    one = np.ones((1, ny, nx))
    if hot:
        near = (x - 0.5) ** 2 + (y - 0.5) ** 2 * (ny > 1) < 0.01
        return p, problems.prim_to_cons(p, one, 0 * one, 0 * one, 0 * one, np.where(near, 300.0, 0.1))
    vy = (-3.0 * np.sign(y - 0.5) if ny > 1 else 0.0) * one
    return p, problems.prim_to_cons(p, one, -3.0 * np.sign(x - 0.5), vy, 0 * one, 0.05 * one)


@pytest.mark.parametrize("nx,ny", [(200, 1), (1100, 1), (60, 50)])
@pytest.mark.parametrize("hot", [True, False])
def test_speeds_that_change(nx, ny, hot):
    from gaukuk_b200.sim import Sim
    p, c = _pulse(nx, ny, hot)
    o = gk_oracle.OracleSim(p, c)
    dts = list(o.run(0.05, 0.05))
    with Sim(p, c, mode="parity") as s:
        t, _, _ = s.advance(0.05)
        assert s.dt_log() == dts and t == o.time
        assert np.array_equal(active(p, s.download()), active(p, o.get_cons()))
