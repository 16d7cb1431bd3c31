"""Ensembles of more tiles than are resident at once: full waves of tiles of the
instances' rows and a last wave whose strips are cut shorter.  Every instance must
equal the same problem run alone (bit for bit in parity mode)."""
import numpy as np
import pytest

from gaukuk_b200 import problems
from helpers import active, rel_linf

pytestmark = pytest.mark.gpu

SIZES = [(300, 260), (257, 333), (126, 512), (640, 96), (65, 47), (380, 201), (249, 250)]


def _resident(threads, mode):  # CTAs of the fused stage on the chip
    return 148 * ((384 if mode == "parity" and threads < 256 else 512) // threads)


@pytest.mark.parametrize("threads,rows,copies", [(128, 16, 3), (64, 16, 3), (256, 5, 3), (128, 7, 2)])
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_full_waves_and_a_cut_tail_equal_solo_runs(threads, rows, copies, mode):
    from gaukuk_b200.ensemble import Ensemble
    from gaukuk_b200.sim import Sim
    inst = [problems.kh(nx, ny=ny, seed=i, half_width=0.2 + 0.005 * i)
            for i, (nx, ny) in enumerate(SIZES * copies)]
    tiles = sum(-(-p.nx // (threads - 4)) * -(-p.ny // rows) for p, _ in inst)
    slots = _resident(threads, mode)
    assert tiles > slots and tiles % slots
    sims = [Sim(p, c, mode=mode) for p, c in inst]
    Ensemble(sims, threads=threads, rows=[rows] * len(sims)).run_steps(3)
    for (p, c), s in zip(inst, sims):
        with Sim(p, c, mode=mode) as solo:
            solo.run_steps(3)
            got, ref = active(p, s.download()), active(p, solo.download())
            if mode == "parity":
                assert s.dt_log() == solo.dt_log() and np.array_equal(got, ref)
            else:
                np.testing.assert_allclose(s.dt_log(), solo.dt_log(), rtol=1e-12)
                assert max(rel_linf(got, ref)) <= 1e-12
