"""The first pass of gk_rk2_step_noalloc: a non-zero z momentum and a CFL speed
that is not finite (a NaN momentum; a NaN energy becomes the pressure floor, as
in the reference's ConsToPrim) are refused with the state untouched, a call after a refusal
is as good as the first, and dtmax limits the step.  Grids of one and of several
CTAs per row and more rows than CTAs.  Collected after the allocating tests."""
import ctypes

import numpy as np
import pytest

from gaukuk_b200 import problems
from test_zz_no_alloc import to_device_layout

pytestmark = pytest.mark.gpu

GK_ERR_NONFINITE, GK_ERR_UNSUPPORTED = -3, -4


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (255, 9), (257, 1300)])
def test_refusals_leave_the_state_and_the_next_call_alone(nx, ny, mode):
    import torch
    from gaukuk_b200 import _lib
    from gaukuk_b200.sim import MODES, _descs
    p, c = problems.kh(nx, ny=ny, seed=4)
    gd, pd = _descs(p, MODES[mode], 0)
    L = _lib.load()
    good = torch.from_numpy(to_device_layout(p, c)).cuda().contiguous()

    def step(state, dtmax):
        dt = ctypes.c_double(-1.0)
        rc = L.gk_rk2_step_noalloc(ctypes.byref(gd), ctypes.byref(pd), ctypes.c_void_p(state.data_ptr()),
                                   dtmax, ctypes.byref(dt), None)
        return rc, dt.value

    first = good.clone()
    rc, dt = step(first, 1e300)
    assert rc == 0 and 0 < dt < 1
    for plane, value, want in ((4, 1e-300, GK_ERR_UNSUPPORTED), (1, float("nan"), GK_ERR_NONFINITE)):
        bad = good.clone()
        bad[plane, p.ng + ny - 1, p.ng + nx - 1] = value
        before = bad.clone()
        assert step(bad, 1e300)[0] == want
        g = p.ng
        same = bad[:, g:g + ny, g:g + nx].cpu().numpy().view(np.int64)
        assert np.array_equal(same, before[:, g:g + ny, g:g + nx].cpu().numpy().view(np.int64))
        again = good.clone()
        rc, dt2 = step(again, 1e300)
        assert rc == 0 and dt2 == dt and torch.equal(again, first)
    half = good.clone()
    rc, dt3 = step(half, 0.5 * dt)
    assert rc == 0 and dt3 == 0.5 * dt
