"""The autotuner's trial steps leave a state as it is, whatever accelerations
an earlier state left behind: they are set anew before the first step."""

import numpy as np
import pytest

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu


def test_stale_accelerations_that_are_not_finite(tmp_path):
    s = B.ethane_liquid(60, seed=241, min_dist=1.6, jitter=0.4)
    a = M.Context(potentials=M.POT_AIREBO)
    a.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    a.run(2, 0.25)
    a.write_state(str(tmp_path / "md"))
    acc = np.fromfile(tmp_path / "md.a").reshape(-1, 3)
    assert acc.shape == s["pos"].shape
    acc[::7] = np.nan
    acc[3::7] = np.inf
    acc.tofile(tmp_path / "md.a")

    def run(ctx):
        ctx.set_state(s["pos"], s["vel"])
        ctx.run(5, 0.25)
        assert ctx.task_mode()[1] > 0.0  # the autotuner ran
        return ctx.get_state()

    b = M.Context(potentials=M.POT_AIREBO)
    assert b.load_state(str(tmp_path / "md"), 2) & M.LOADED_A
    got = run(b)
    c = M.Context(potentials=M.POT_AIREBO)
    c.load_state(str(tmp_path / "md"), 0)  # (iteration 0: the accelerations are not taken)
    want = run(c)
    # the splits may differ between the two, and agree to rounding
    assert np.allclose(got[0], want[0], rtol=0, atol=1e-9) and np.allclose(got[1], want[1], rtol=0, atol=1e-9)
    assert np.array_equal(got[2], want[2])
