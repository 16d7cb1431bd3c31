"""Sides that bring z momentum into a 1D or 2D run that has none: fixed data and a
host routine.  A massless point mass (its kicks add zeros) puts the same problem
among the runs that carry v_z from the start; state and dt sequence must be its
bits.  The z speed of the inflow soon sets dt."""
import ctypes

import numpy as np
import pytest

from gaukuk_b200 import _lib, problems
from gaukuk_b200.config import Params
from helpers import active

pytestmark = pytest.mark.gpu

FILL = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p)


@pytest.mark.parametrize("nx,ny", [(64, 1), (1100, 1), (40, 24)])
@pytest.mark.parametrize("integrator", [2, 3])
@pytest.mark.parametrize("how", ["fixed", "host"])
def test_inflow_of_z_momentum(nx, ny, integrator, how):
    from gaukuk_b200.sim import Sim
    p = Params(nx=nx, ny=ny, bc=(4 if how == "fixed" else 0, 3, 2, 3, 1, 1), integrator=integrator,
               tmax=10.0, dtoutput=10.0, stepmax=30)
    c = problems.random_smooth(p, seed=3)
    assert not c[3].any()
    inflow = c.copy()
    left = inflow[:, p.ng, :, :p.ng]
    left[:] = np.array([1.0, 2.0, 0.0, 12.0, 80.0])[:, None, None]
    host = np.zeros_like(c)

    def fill(_, __):
        host[:, p.ng, p.ng:p.ng + ny, :p.ng] = left[:, p.ng:p.ng + ny]
        return 0
    fn = FILL(fill)
    out = []
    for mass in ([], [(0.0, 0.5, 0.5, 0.5, 0.3)]):
        with Sim(p, c, mode="parity") as s:
            s.set_point_gravity(mass)
            if how == "fixed":
                s.set_fixed_boundary(inflow)
            else:
                _lib.check(_lib.load().gk_set_host_fill(s.h, 0, 1, ctypes.cast(fn, ctypes.c_void_p), None,
                                                        host.ctypes.data_as(ctypes.c_void_p)), s.h)
            s.run()
            out.append((active(p, s.download()).copy(), s.dt_log()))
    (a, da), (b, db) = out
    assert b[3].any()
    assert da == db and np.array_equal(a, b)
