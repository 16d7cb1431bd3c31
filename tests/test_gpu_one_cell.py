"""A grid of one cell, whose ghosts are copied from ghosts: every pair of x sides
against the oracle, which fills them in the reference's order and swaps its
arrays after every step."""
import numpy as np
import pytest

import gk_oracle
from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [0, 1, 2, 3])
@pytest.mark.parametrize("right", [0, 1, 2, 3])
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_one_cell_equals_the_oracle(left, right, mode):
    from gaukuk_b200.sim import Sim
    one = np.ones((1, 1, 1))
    for integrator, rc_order, grav, vx in ((1, 2, 0.0, 0.3), (2, 2, 0.0, -0.4), (2, 1, 0.2, 0.3), (3, 2, 0.0, 0.3),
                                           (3, 2, -0.3, 0.1)):
        p = Params(nx=1, bc=(left, right, 1, 1, 1, 1), integrator=integrator, rc_order=rc_order,
                   grav=(grav, 0.0, 0.0), tmax=10.0, dtoutput=10.0, stepmax=6)
        c = problems.prim_to_cons(p, 1.3 * one, vx * one, 0 * one, 0 * one, 0.8 * one)
        o = gk_oracle.OracleSim(p, c)
        dts = o.run(p.tmax, p.dtoutput)
        ref = active(p, o.get_cons())
        with Sim(p, c, mode=mode) as s:
            s.run(p.tmax, p.dtoutput)
            got = active(p, s.download())
            if mode == "parity":
                assert s.dt_log() == dts and np.array_equal(got, ref)
            else:
                np.testing.assert_allclose(s.dt_log(), dts, rtol=1e-12)
                assert np.abs(got - ref).max() <= 1e-12  # of values about 1
