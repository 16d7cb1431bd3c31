"""The ghost strips of a downloaded frame are the fill of the last stage state
of the steps that ran, whatever path the handle has taken since: a change of
path, or a run that takes no step on the new path, leaves the frame as it is."""
import numpy as np
import pytest

from gaukuk_b200 import learned, problems
from gaukuk_b200.config import Params

pytestmark = pytest.mark.gpu


def _problem(nx, ny, vz, integrator, stepmax=0):
    p = Params(nx=nx, ny=ny, bc=(1, 1, 2, 3, 1, 1), integrator=integrator, tmax=1.0, dtoutput=1.0,
               stepmax=stepmax)
    return p, problems.random_smooth(p, seed=nx + ny, with_vz=vz)


def _install(s, fused):
    blob = np.zeros(learned.NMODEL, dtype=np.float32)  # adds zeros
    blob[learned.NPARAM + 16:learned.NPARAM + 32] = 1.0
    blob[learned.NPARAM + 36:] = 1.0
    learned.install(s, blob, fused=fused)


def _mass(s):
    s.set_point_gravity([(0.0, 0.5, 0.5, 0.5, 0.3)])


# problem, how the handle starts, how its path changes
CHANGES = {
    "short_row": ((200, 1, False), None, _mass),
    "fused2d_to_five": ((61, 40, False), None, _mass),
    "fused2d_to_pass": ((61, 40, False), None, lambda s: _install(s, False)),
    "five_to_pass": ((61, 40, True), None, lambda s: _install(s, False)),
    "pass_to_five": ((61, 40, True), lambda s: _install(s, False), lambda s: learned.install(s, None)),
    "pass_to_learned_stage": ((61, 40, False), lambda s: _install(s, False), lambda s: _install(s, True)),
}


@pytest.mark.parametrize("integrator", [1, 2, 3])
@pytest.mark.parametrize("name", sorted(CHANGES))
def test_a_change_of_path_leaves_the_frame(name, integrator):
    from gaukuk_b200.sim import Sim
    (nx, ny, vz), start, change = CHANGES[name]
    p, c = _problem(nx, ny, vz, integrator, stepmax=3)
    with Sim(p, c, mode="parity") as s:
        if start:
            start(s)
        s.run_steps(2)
        want = s.download()
        change(s)
        assert np.array_equal(s.download(), want)
        s.run_steps(1)
        want = s.download()
    # the last step on the new path alone, from the same state
    with Sim(p, c, mode="parity") as s:
        if start:
            start(s)
        s.run_steps(2)
        change(s)
        s.run_steps(1)
        assert np.array_equal(s.download(), want)
        # no step is left: a run on the first path takes none
        if start:
            start(s)
        elif change is _mass:
            s.set_point_gravity([])
        else:
            learned.install(s, None)
        assert s.run_steps(1) == 0
        assert np.array_equal(s.download(), want)


@pytest.mark.parametrize("integrator", [2, 3])
def test_paths_leave_the_same_strips(integrator):
    """Steps on the short-row path and then on the row stage: the strips of the
    row stage alone, run from the start."""
    from gaukuk_b200.sim import Sim
    p, c = _problem(200, 1, False, integrator)
    out = []
    for before in (2, 0):
        with Sim(p, c, mode="parity") as s:
            s.run_steps(before)
            _mass(s)
            s.run_steps(3 - before)
            out.append(s.download())
    assert np.array_equal(*out)
