"""Gravity along z in 1D and 2D runs that start with no z momentum: the kicks make
one, which the CFL speed counts.  State and dt sequence against the oracle; the
z speed soon sets dt.  The first kick moves the momentum at rest without the
energy, so that coarse grids start at the pressure floor: a pressure left over
from two kinetic energies is rounding, and with it fast mode's state (two cells:
4 floor hits in the first step, mass fluxes 1e-9 apart).  There fast mode is held
to the dt sequence."""
import numpy as np
import pytest

import gk_oracle
from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active, rel_linf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 1), (64, 1), (1100, 1), (33, 20)])
@pytest.mark.parametrize("integrator", [1, 2, 3])
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_z_gravity_from_rest(nx, ny, integrator, mode):
    from gaukuk_b200.sim import Sim
    p = Params(nx=nx, ny=ny, bc=(1, 1, 2, 3, 1, 1), integrator=integrator, grav=(0.0, 0.0, 200.0),
               tmax=10.0, dtoutput=10.0, stepmax=40)
    c = problems.random_smooth(p, seed=nx)
    assert not c[3].any()
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
            assert s.floor_hits()[1] or max(rel_linf(got, ref)) <= 1e-12
