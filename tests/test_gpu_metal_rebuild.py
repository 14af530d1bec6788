"""The metal and ion list is rebuilt in every launch configuration: an ion that
has moved further than the list's skin meets the atoms it has come to, so the
last step's energy is that of the final positions evaluated afresh."""
import numpy as np
import pytest

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("task_mode", [0, 2])
def test_ion_path_rebuilds_the_metal_list(task_mode):
    s = B.fcc(29, 8, 8, 4, pbc=(1, 1, 0), temp_k=300.0, seed=9)
    top, edge = s["pos"][:, 2].max(), s["box"][0]
    mol = B.c2h6_example()
    s = B.add_atoms(s, mol["z"], mol["pos"] - mol["pos"].mean(axis=0) + [6.0, 6.0, top + 3.0])
    # beyond the list range (7.92 A) at first, 4 A above the surface at the end
    s = B.add_atoms(s, [18], [[edge * 0.7, edge * 0.7, top + 9.0]], vel=[[0.0, 0.0, -0.25]])
    ctx = M.Context(potentials=M.POT_AIREBO | M.POT_METAL, task_mode=task_mode)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    epot, _ = ctx.run(80, 0.25)
    pos, vel, _ = ctx.get_state()
    fresh = M.Context(potentials=M.POT_AIREBO | M.POT_METAL, task_mode=task_mode)
    fresh.set_system(s["z"], pos, vel, s["box"], s["pbc"], s["fixed"])
    e, terms, _ = fresh.compute()
    assert abs(terms[3]) > 1.0
    # the two sums differ in order only
    assert abs(epot[-1] - e) <= 1e-11 * abs(e)
