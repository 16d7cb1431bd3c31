"""The fused 2D stage in tiles (small grids) against the oracle and against the
marching kernels, at the edges of its tiles: 28 columns, 4 or 10 rows, one and
several tiles per CTA."""
import numpy as np
import pytest

import gk_oracle
from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active, rel_linf

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (28, 4), (29, 5), (27, 41), (57, 10), (56, 11), (113, 3), (300, 170)]


def _problem(nx, ny, bc, integrator, grav, rc_order):
    p = Params(nx=nx, ny=ny, bc=bc + (1, 1), integrator=integrator, grav=grav, rc_order=rc_order, tmax=1.0,
               dtoutput=1.0, stepmax=3)
    return p, problems.random_smooth(p, seed=nx + ny)


@pytest.mark.parametrize("rows", ["4", "10"])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_tiles_equal_the_oracle_and_the_marching_stage(nx, ny, rows, monkeypatch):
    from gaukuk_b200.sim import Sim
    for bc, integrator, grav, rc_order in (((1, 1, 1, 1), 2, (0, 0, 0), 2), ((1, 1, 2, 2), 3, (0.1, -0.2, 0), 2),
                                           ((0, 3, 3, 2), 2, (0, 0, 0), 1)):
        p, c = _problem(nx, ny, bc, integrator, grav, rc_order)
        o = gk_oracle.OracleSim(p, c)
        dts = o.run(p.tmax, p.dtoutput)
        out = {}
        for mode in ("parity", "fast"):
            for tile in (rows, "0"):
                monkeypatch.setenv("GK_STAGE_TILE", tile)
                with Sim(p, c, mode=mode) as s:
                    assert s.path == "fused2d"
                    s.run(p.tmax, p.dtoutput)
                    out[mode, tile] = s.download()
                    if mode == "parity":
                        assert s.dt_log() == dts
        assert np.array_equal(active(p, out["parity", rows]), active(p, o.get_cons()))
        assert np.array_equal(out["parity", rows], out["parity", "0"])  # ghosts too
        assert max(rel_linf(active(p, out["fast", rows]), active(p, out["fast", "0"]))) <= 1e-12
