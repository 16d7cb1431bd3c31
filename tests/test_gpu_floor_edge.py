"""Pressures between zero and their floor, and next to it, in every kernel that
tests the floor: the hits of fast mode are parity mode's.

A uniform flow whose cells carry less energy than the pressure floor asks for
has uniform primitives (the conversion floors them), so its fluxes cancel and
each stage meets the cell's own pressure again: a cell below the floor is
counted once per stage, a cell above it never."""
import ctypes
import dataclasses

import numpy as np
import pytest

from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active, rel_linf

pytestmark = pytest.mark.gpu

# pressure over its floor; the nearest are 1e-13 away, rounding is at 1e-15
BELOW = (0.0, 0.1, 0.5, 1 - 1e-6, 1 - 1e-9, 1 - 1e-11, 1 - 1e-12, 1 - 1e-13)
ABOVE = (1 + 1e-13, 1 + 1e-12, 1 + 1e-11, 1 + 1e-9)


def _state(nx, ny, nz, vz, integrator, seed=0):
    p = Params(nx=nx, ny=ny, nz=nz, integrator=integrator, bc=(1,) * 6, pfloor=0.05, tmax=1.0, dtoutput=1.0,
               stepmax=1)
    sh = (nz, ny, nx)
    one = np.ones(sh)
    c = problems.prim_to_cons(p, one, 0.4 * one, -0.3 * one, vz * one, p.pfloor * one)
    rng = np.random.default_rng(nx * ny + seed)
    of = rng.choice(BELOW, sh)
    # a few cells above the floor, 16 apart, and no near ones within their reach
    for at in np.argwhere(np.ones([max(1, n // 16) for n in sh])) * 16:
        away = [np.minimum((np.arange(n) - m) % n, (m - np.arange(n)) % n) for n, m in zip(sh, at)]
        of[np.ix_(*[d <= 6 for d in away])] = 0.5
    for at in np.argwhere(np.ones([max(1, n // 16) for n in sh])) * 16:
        of[tuple(at)] = rng.choice(ABOVE)
    a = active(p, c)
    a[4] += (of - 1) * p.pfloor / (p.gamma - 1)
    return p, c, int((of < 1).sum())


# the fused 2D stage in tiles of 4 and 10 rows, marching by TMA and by plain
# loads; five variables in 2D; 3D
KERNELS = {"tiles4": (93, 61, 1, 0.0, {"GK_STAGE_TILE": "4"}),
           "tiles10": (93, 61, 1, 0.0, {"GK_STAGE_TILE": "10"}),
           "tma": (131, 50, 1, 0.0, {"GK_STAGE_TILE": "0"}),
           "loads": (131, 50, 1, 0.0, {"GK_STAGE_TILE": "0", "GK_STAGE_TMA": "0"}),
           "five": (61, 17, 1, 0.2, {}),
           "3d": (21, 18, 9, 0.2, {}),
           "row": (1100, 1, 1, 0.0, {}),
           "short_row": (257, 1, 1, 0.0, {})}


@pytest.mark.parametrize("integrator", [2, 3])
@pytest.mark.parametrize("kernel", sorted(KERNELS))
def test_hits_per_stage(kernel, integrator, monkeypatch):
    from gaukuk_b200.sim import Sim
    nx, ny, nz, vz, env = KERNELS[kernel]
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    p, c, below = _state(nx, ny, nz, vz, integrator)
    out = []
    for mode in ("parity", "fast"):
        with Sim(p, c, mode=mode) as s:
            s.run(p.tmax, p.dtoutput)
            out.append((active(p, s.download()), s.floor_hits(), s.dt_log()))
    (a, ha, da), (b, hb, db) = out
    assert ha == (0, integrator * below)
    assert hb == ha
    np.testing.assert_allclose(db, da, rtol=1e-12)
    assert max(rel_linf(b, a)) <= 1e-12


@pytest.mark.parametrize("kick", ["gravity", "point"])
def test_last_stage_with_a_kick_in_3d(kick):
    from gaukuk_b200.sim import Sim
    p, c, _ = _state(21, 18, 9, 0.2, 2)
    if kick == "gravity":
        p = dataclasses.replace(p, grav=(0.01, 0.0, 0.02))
    out = []
    for mode in ("parity", "fast"):
        with Sim(p, c, mode=mode) as s:
            if kick == "point":
                s.set_point_gravity([(0.01, 0.4, 0.6, 0.5, 0.3)])
            s.run(p.tmax, p.dtoutput)
            out.append(active(p, s.download()))
    assert max(rel_linf(out[1], out[0])) <= 1e-12


def test_ensemble():
    from gaukuk_b200.ensemble import Ensemble
    from gaukuk_b200.sim import Sim
    inst = [_state(61, 40, 1, 0.0, 2, seed=i) for i in range(3)]
    out = []
    for mode in ("parity", "fast"):
        sims = [Sim(p, c, mode=mode) for p, c, _ in inst]
        Ensemble(sims).run_steps(1)
        out.append([(active(p, s.download()), s.floor_hits()) for s, (p, _, _) in zip(sims, inst)])
    for (a, ha), (b, hb), (_, _, below) in zip(*out, inst):
        assert ha == hb == (0, 2 * below)
        assert max(rel_linf(b, a)) <= 1e-12


def test_step_on_a_device_array():
    """A flow that expands to below the floor in the first stage only: what the
    floor adds there stays in the new state."""
    import torch
    from gaukuk_b200 import _lib
    from gaukuk_b200.sim import MODES, Sim, _descs
    p = Params(nx=130, ny=94, bc=(1,) * 6, integrator=2, pfloor=0.05, tmax=1.0, dtoutput=1.0)
    rng = np.random.default_rng(8)
    sh = (1, p.ny, p.nx)
    x = np.arange(p.nx)[None, None, :] / p.nx
    c = problems.prim_to_cons(p, np.ones(sh), np.sin(20 * np.pi * x) * np.ones(sh), rng.uniform(-0.3, 0.3, sh),
                              np.zeros(sh), p.pfloor * rng.uniform(1.0, 1.2, sh))
    pitch = (p.lenx + 15) // 16 * 16
    u = np.zeros((5, p.leny, pitch))
    for slot, v in enumerate((0, 1, 2, 4, 3)):
        u[slot, :, :p.lenx] = c[v, p.ng]
    with Sim(p, c, mode="parity") as s:
        s.run_steps(1)
        want = active(p, s.download())[:, 0]
        assert s.floor_hits()[1] > 100
    gd, pd = _descs(p, MODES["fast"], 0)
    state, dt = torch.from_numpy(u).cuda(), ctypes.c_double()
    _lib.check(_lib.load().gk_rk2_step_noalloc(ctypes.byref(gd), ctypes.byref(pd),
                                               ctypes.c_void_p(state.data_ptr()), 1e300, ctypes.byref(dt), None))
    got = state.cpu().numpy()[:, p.ng:p.ng + p.ny, p.ng:p.ng + p.nx]
    for slot, v in enumerate((0, 1, 2, 4)):
        assert np.abs(got[slot] - want[v]).max() <= 1e-12 * np.abs(want[v]).max()
