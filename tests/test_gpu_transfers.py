"""Whole-state transfers: what comes back is what went up, and after a step the
ghost strips are the fill of the last stage state.

The strips of a periodic RK2 run after one step are the wrap of its stage-1
state, which is the state a forward Euler run reaches in one step (same dt);
every other stored ghost keeps its uploaded value.  Sizes: one, two and three
directions, uneven, on each path that has its own transfer."""
import numpy as np
import pytest

from gaukuk_b200 import problems
from gaukuk_b200.config import Params
from helpers import active

pytestmark = pytest.mark.gpu

SHAPES = {"run1d": (37, 1, 1), "row": (1031, 1, 1), "fused2d": (19, 23, 1), "fused2d_wide": (131, 2, 1),
          "generic2d": (18, 27, 1), "stage3d": (9, 7, 5), "stage3d_flat": (33, 3, 2)}


def _random(p, vz):
    rng = np.random.default_rng(11)
    sh = (p.nz, p.ny, p.nx)
    v = [rng.uniform(-0.5, 0.5, sh) for _ in range(3)]
    c = problems.prim_to_cons(p, rng.uniform(1, 2, sh), v[0], v[1] if p.ny > 1 else 0 * v[1],
                              v[2] if vz else 0 * v[2], rng.uniform(1, 2, sh))
    stored = slice(None) if p.nz > 1 else slice(p.ng, p.ng + 1)
    edge = np.ones(c.shape, dtype=bool)
    active(p, edge)[...] = False
    if p.nz == 1 and not vz:
        edge[3] = False  # a zero z momentum keeps 2D runs on the fused path
    c[edge] = rng.uniform(1, 2, int(edge.sum()))
    return c, stored


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("planes_only", [False, True])
def test_round_trip_and_strips(name, planes_only):
    from gaukuk_b200.sim import Sim
    nx, ny, nz = SHAPES[name]
    vz = nz > 1 or name == "generic2d"
    p = Params(nx=nx, ny=ny, nz=nz, bc=(1,) * 6, integrator=2, tmax=1.0, dtoutput=1.0)
    c, stored = _random(p, vz)
    with Sim(p, c, mode="parity") as s:
        got = s.download()
        assert np.array_equal(got[:, stored], c[:, stored])
        if nz == 1:
            got[:, stored] = 0
            assert not got.any()
        s.run_steps(1)
        out = c.copy()
        got = s.download(out, planes_only=planes_only)
        if planes_only and nz == 1:
            other = [k for k in range(p.lenz) if k != p.ng]
            assert np.array_equal(got[:, other], c[:, other])
        new = active(p, got).copy()
    e = Params(**{**p.__dict__, "integrator": 1})
    with Sim(e, c, mode="parity") as s:
        s.run_steps(1)
        u1 = active(e, s.download()).copy()
    want = c[:, stored].copy()
    g, kz = p.ng, (p.ng if nz > 1 else 0)
    act = [slice(kz, kz + nz), slice(g, g + ny), slice(g, g + nx)]
    for ax, n in ((2, nx), (1, ny), (0, nz)):
        if n == 1:
            continue
        for q in range(g):
            for dst, src in ((q, n - g + q), (g + n + q, q)):
                d, f = list(act), [slice(None)] * 3
                d[ax], f[ax] = dst, src
                want[(slice(None), *d)] = u1[(slice(None), *f)]
    want[(slice(None), *act)] = new
    if name.startswith("fused2d"):
        want[3] = got[:, stored][3]  # MTZ: zero at upload, left alone
    assert np.array_equal(got[:, stored], want)
