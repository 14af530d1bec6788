"""Brenner by bond ends against the per-atom kernel.  A bond capacity of 1,100
puts the bond records beyond their limit, so the per-atom kernel runs.  Both
add the same terms in other orders; the tables' monomials in absolute
coordinates sum terms of up to 1e6 times their value, so 2e-16 of rounding in
an argument becomes at most about 2e-10 of a force."""
import numpy as np
import pytest

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "molecule": lambda: B.c2h6_example(),
    "diamond": lambda: B.diamond(3, disp_sigma=0.15, seed=51),
    "amorphous": lambda: B.amorphous_carbon(250, h_fraction=0.3, seed=52),
    "hydrogen": lambda: B.amorphous_carbon(60, h_fraction=1.0, density_g_cm3=0.2, min_sep=0.9, seed=53),
    "dense": lambda: B.amorphous_carbon(300, density_g_cm3=2.6, min_sep=1.2, seed=54),
}


def _force(s, pot, brenner_set, **kw):
    ctx = M.Context(potentials=pot, brenner_set=brenner_set, **kw)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    out = ctx.compute()
    ctx.close()
    return out


@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("brenner_set", [1, 2])
@pytest.mark.parametrize("tors", [0, M.POT_ETORS])
def test_bond_ends_equal_per_atom_kernel(name, brenner_set, tors):
    s = SYSTEMS[name]()
    a = _force(s, M.POT_BRENNER | tors, brenner_set)
    b = _force(s, M.POT_BRENNER | tors, brenner_set, cap_bonds=1100)
    assert abs(a[0] - b[0]) <= 1e-10 * abs(b[0])
    assert np.all(np.abs(a[1] - b[1]) <= 1e-10 * abs(b[0]))
    assert np.linalg.norm(a[2] - b[2]) <= 1e-9 * np.linalg.norm(b[2])
