"""Which Brenner kernel a context takes, and that both give the same forces.

The bond-end kernel keeps a record per bond slot, sized for every slot in use;
the per-atom kernel keeps none.  Beyond 8e9 bytes of records, or when they
would leave less memory free than they take, the per-atom kernel runs.  Both
add the same terms in other orders; the tables' monomials in absolute
coordinates sum terms of up to 1e6 times their value, so 2e-16 of rounding in
an argument becomes at most about 2e-10 of a force."""
import numpy as np
import pytest
import torch

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

# a bond capacity for each size that puts n cap (5 + 4 cap) 8 bytes above 8e9
SYSTEMS = {
    "molecule": (lambda: B.c2h6_example(), 5650),
    "hydrogen": (lambda: B.amorphous_carbon(60, h_fraction=1.0, density_g_cm3=0.2, min_sep=0.9, seed=53), 2080),
}


def _force(s, pot, brenner_set, **kw):
    """(energies and gradient, the kernels that ran)"""
    ctx = M.Context(potentials=pot, brenner_set=brenner_set, **kw)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    ctx.set_profiling(True)
    out = ctx.compute()
    kernels = ctx.profile_read()
    ctx.close()
    return out, set(kernels)


def _same(a, b):
    assert abs(a[0] - b[0]) <= 1e-10 * abs(b[0])
    assert np.all(np.abs(a[1] - b[1]) <= 1e-10 * abs(b[0]))
    assert np.linalg.norm(a[2] - b[2]) <= 1e-9 * np.linalg.norm(b[2])


@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("brenner_set", [1, 2])
@pytest.mark.parametrize("tors", [0, M.POT_ETORS])
def test_small_systems_on_both_kernels(name, brenner_set, tors):
    build, cap = SYSTEMS[name]
    s = build()
    assert len(s["z"]) * cap * (5 + 4 * cap) * 8 > 8e9
    a, ka = _force(s, M.POT_BRENNER | tors, brenner_set)
    b, kb = _force(s, M.POT_BRENNER | tors, brenner_set, cap_bonds=cap)
    assert "bond_reduce" in ka and "bond_reduce" not in kb  # the sums of the bond-end kernel's records
    _same(a, b)


def test_records_that_do_not_fit_are_not_required():
    """A GPU with 3 GB left loads a system whose records would take 7.9 GB."""
    s = B.diamond(3, disp_sigma=0.15, seed=51)
    cap = 1070
    assert 7.8e9 < len(s["z"]) * cap * (5 + 4 * cap) * 8 < 8e9
    a, ka = _force(s, M.POT_BRENNER, 1, cap_bonds=cap)
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - 3 * 10**9, dtype=torch.uint8, device="cuda")
    try:
        b, kb = _force(s, M.POT_BRENNER, 1, cap_bonds=cap)
    finally:
        del held
        torch.cuda.empty_cache()
    assert "bond_reduce" in ka and "bond_reduce" not in kb
    _same(a, b)
