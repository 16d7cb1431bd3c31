"""Slabs on the marching forms of the fused 2D stage, which grids of this size take
only when told to: with rows staged by TMA and by plain loads the split grid still
takes one step where the undivided one does, bit for bit."""
import dataclasses

import numpy as np
import pytest

from gaukuk_b200 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tma", ["1", "0"])
@pytest.mark.parametrize("integrator", [2, 3])
def test_slabs_on_the_marching_stage(tma, integrator, monkeypatch):
    from gaukuk_b200.sim import Sim
    from gaukuk_b200.slabs import Slabs
    monkeypatch.setenv("GK_STAGE_TILE", "0")
    monkeypatch.setenv("GK_STAGE_TMA", tma)
    p, c = problems.kh(160, ny=150, seed=3)
    p = dataclasses.replace(p, integrator=integrator, tmax=0.2, dtoutput=0.05, stepmax=20)
    with Sim(p, c, mode="parity") as s:
        s.run(p.tmax, p.dtoutput)
        want, want_dts = s.download(), s.dt_log()
    with Slabs(p, c, 3, mode="parity") as s:
        s.run(p.tmax, p.dtoutput)
        assert s.dt_log() == want_dts
        assert np.array_equal(s.download(), want)
