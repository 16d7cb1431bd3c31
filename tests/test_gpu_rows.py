"""The 1D row stage (path 0): against the oracle at the edges of its tiles (124
cells, one tile per CTA up to 444 of them) and against the path of short rows
(path 3, in one CTA or a cluster), whole frames with their ghosts, on every pair
of x sides."""
import numpy as np
import pytest

import gk_oracle
from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active

pytestmark = pytest.mark.gpu


def _problem(nx, bc, integrator, rc_order=2, grav=0.0):
    p = Params(nx=nx, bc=(bc[0], bc[1], 1, 1, 1, 1), integrator=integrator, rc_order=rc_order,
               grav=(grav, 0.0, 0.0), tmax=1.0, dtoutput=1.0, stepmax=3)
    rng = np.random.default_rng(nx)
    sh = (1, 1, nx)
    v = rng.uniform(-1, 1, sh)
    return p, problems.prim_to_cons(p, rng.uniform(0.5, 2, sh), v, np.zeros(sh), np.zeros(sh),
                                    rng.uniform(0.5, 2, sh))


# (grid of 444 CTAs: 55056 cells fill it once)
@pytest.mark.parametrize("nx,grav", [(2, 0.1), (5, -0.1), (124, 0.1), (125, 0.1), (1021, 0.0), (1240, 0.0),
                                     (1241, 0.1), (55056, 0.0), (55057, 0.0), (120001, 0.0)])
@pytest.mark.parametrize("integrator", [2, 3])
def test_rows_equal_the_oracle(nx, grav, integrator):
    from gaukuk_b200.sim import Sim
    p, c = _problem(nx, (2, 3), integrator, grav=grav)
    o = gk_oracle.OracleSim(p, c)
    dts = o.run(p.tmax, p.dtoutput)
    with Sim(p, c, mode="parity") as s:
        assert s.path == "generic"
        s.run(p.tmax, p.dtoutput)
        assert s.dt_log() == dts
        assert np.array_equal(active(p, s.download()), active(p, o.get_cons()))


@pytest.mark.parametrize("left", [0, 1, 2, 3])
@pytest.mark.parametrize("right", [0, 1, 2, 3])
def test_rows_equal_the_short_row_path(left, right, monkeypatch):
    from gaukuk_b200.sim import Sim
    # one CTA up to 316 cells, then 3 to 8 CTAs in a cluster
    for nx, integrator, rc_order in ((2, 2, 2), (3, 3, 2), (248, 2, 2), (316, 3, 1), (317, 2, 2), (385, 1, 2),
                                     (640, 3, 2), (1020, 2, 2), (1020, 3, 1)):
        p, c = _problem(nx, (left, right), integrator, rc_order)
        out = []
        for run1d in ("1", "0"):
            monkeypatch.setenv("GK_RUN1D", run1d)
            with Sim(p, c, mode="parity") as s:
                assert s.path == ("run1d" if run1d == "1" else "generic")
                s.run(p.tmax, p.dtoutput)
                out.append((s.download(), s.dt_log()))
        (a, da), (b, db) = out
        assert da == db
        assert np.array_equal(a, b)
