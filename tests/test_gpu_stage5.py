"""2D runs with five evolved variables: the one-launch stage against the
per-phase kernels it replaces.

The per-phase kernels still run for a handle with the learned correction as a
pass; with a zero model that pass adds zeros, so both must give the same bits
in parity mode, dt sequence included, and agree to 1e-12 in fast mode.  Sizes
at the edges of the CTA's columns (60 and 124 updated) and of its rows; kicks
of constant gravity, one point mass and a binary."""
import numpy as np
import pytest

from gaukuk_b200 import learned, problems
from gaukuk_b200.config import Params
from helpers import active, rel_linf

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (60, 3), (61, 17), (124, 2), (125, 33), (131, 70)]
KICKS = {"none": ((0, 0, 0), []), "gravity": ((0.1, -0.2, 0.3), []),
         "point": ((0, 0, 0), [(0.5, 0.4, 0.6, 0.1, 0.3)]),
         "binary": ((0, 0.1, 0), [(0.5, 0.4, 0.6, 0.0, 0.3), (0.2, 0.9, 0.5, 0.0, 0.2)])}


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("kick", sorted(KICKS))
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_stage_is_the_phase_kernels(nx, ny, kick, mode):
    from gaukuk_b200.sim import Sim
    grav, masses = KICKS[kick]
    for integrator, rc_order in ((2, 2), (3, 2), (2, 1)):
        p = Params(nx=nx, ny=ny, bc=(1, 1, 2, 3, 1, 1), integrator=integrator, rc_order=rc_order,
                   grav=grav, tmax=1.0, dtoutput=1.0)
        c = problems.random_smooth(p, seed=nx, with_vz=True)
        out = []
        for passes in (False, True):
            with Sim(p, c, mode=mode) as s:
                s.set_point_gravity(masses)
                if passes:
                    blob = np.zeros(learned.NMODEL, dtype=np.float32)
                    blob[learned.NPARAM + 16:learned.NPARAM + 32] = 1.0
                    blob[learned.NPARAM + 36:] = 1.0
                    learned.install(s, blob, fused=False)
                assert s.path == "generic"
                s.run_steps(4)
                out.append((active(p, s.download()).copy(), s.dt_log()))
        (a, da), (b, db) = out
        if mode == "parity":
            assert da == db and np.array_equal(a, b)
        else:
            assert max(rel_linf(a, b)) <= 1e-12
            assert np.allclose(da, db, rtol=1e-12, atol=0)
