"""Fast mode's floors (the test without a reciprocal in stages that take no CFL
speed, and the pressure the last stage hands to the CFL speed) against parity
mode's, and long 1D rows around the sizes where the stage launch changes."""
import numpy as np
import pytest

import gk_oracle
from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active, rel_linf

pytestmark = pytest.mark.gpu


def _floored(nx, ny, nz, integrator):
    """Uniform flow whose every 7th cell has far too little energy and every
    53rd far too little density."""
    p = Params(nx=nx, ny=ny, nz=nz, integrator=integrator, bc=(1,) * 6, dfloor=1e-2, pfloor=1e-3, tmax=1.0,
               dtoutput=1.0, stepmax=2)
    rng = np.random.default_rng(nx + ny)
    sh = (nz, ny, nx)
    one = np.ones(sh)
    c = problems.prim_to_cons(p, one, 0.4 * one, -0.3 * one, (0.2 if nz > 1 else 0.0) * one,
                              rng.uniform(0.8, 1.2, sh))
    a = active(p, c)
    flat = a.reshape(5, -1)
    flat[4, ::7] -= rng.uniform(3.0, 4.0, flat[4, ::7].shape)
    flat[0, ::53] = 1e-3
    flat[1:4, ::53] = 0.0
    a[...] = flat.reshape(a.shape)
    return p, c


# 2D: in tiles of 4 and 10 rows and by the marching kernel; 3D
@pytest.mark.parametrize("nx,ny,nz,tile", [(93, 61, 1, "4"), (93, 61, 1, "10"), (131, 50, 1, "0"), (21, 18, 9, "0")])
@pytest.mark.parametrize("integrator", [2, 3])
def test_floors_hit_the_same_cells_in_both_modes(nx, ny, nz, tile, integrator, monkeypatch):
    from gaukuk_b200.sim import Sim
    monkeypatch.setenv("GK_STAGE_TILE", tile)
    p, c = _floored(nx, ny, nz, integrator)
    out = []
    for mode in ("parity", "fast"):
        with Sim(p, c, mode=mode) as s:
            s.run(p.tmax, p.dtoutput)
            out.append((active(p, s.download()), s.floor_hits(), s.dt_log()))
    (a, ha, da), (b, hb, db) = out
    assert ha == hb and ha[0] > 0 and ha[1] > 0
    np.testing.assert_allclose(db, da, rtol=1e-12)
    assert max(rel_linf(b, a)) <= 1e-12


# 124 cells per tile: three CTAs per SM up to 444 tiles, then four (parity) or five (fast)
@pytest.mark.parametrize("mode,nx", [("parity", 55057), ("parity", 73408), ("parity", 73409), ("fast", 55056),
                                     ("fast", 55057), ("fast", 91760), ("fast", 91761)])
def test_long_rows(mode, nx):
    from gaukuk_b200.sim import Sim
    p = Params(nx=nx, bc=(2, 3, 1, 1, 1, 1), integrator=2, tmax=1.0, dtoutput=1.0, stepmax=3)
    rng = np.random.default_rng(nx)
    sh = (1, 1, nx)
    c = problems.prim_to_cons(p, rng.uniform(0.5, 2, sh), rng.uniform(-1, 1, sh), np.zeros(sh), np.zeros(sh),
                              rng.uniform(0.5, 2, sh))
    o = gk_oracle.OracleSim(p, c)
    dts = o.run(p.tmax, p.dtoutput)
    with Sim(p, c, mode=mode) as s:
        assert s.path == "generic"
        s.run(p.tmax, p.dtoutput)
        got, ref = active(p, s.download()), active(p, o.get_cons())
        if mode == "parity":
            assert s.dt_log() == dts and np.array_equal(got, ref)
        else:
            np.testing.assert_allclose(s.dt_log(), dts, rtol=1e-12)
            assert max(rel_linf(got, ref)) <= 1e-12
