"""The connectivity table built by groups of lanes against the one-thread
build.  A bond capacity above 32 sends every atom to the one-thread build; the
tables, and with them every LJ pair's class, weight and path, must be the same,
so energies and gradients agree bit for bit."""
import numpy as np
import pytest

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

SYSTEMS = {
    # few candidates; a remainder of the group; a group's worth of 2-bond paths and twice that
    "molecule": lambda: B.c2h6_example(),
    "ethane_odd": lambda: B.ethane_liquid(29, seed=41),
    "graphite": lambda: B.graphite_slab(2, 5, 3, temp_k=2000.0, seed=42),
    "diamond": lambda: B.diamond(4, disp_sigma=0.12, seed=43),
    # equal weights met on several paths (every cutoff 1)
    "diamond_perfect": lambda: B.diamond(4, seed=44),
    # more candidates than a row holds for some atoms, fewer for others
    "dense": lambda: B.amorphous_carbon(400, density_g_cm3=2.6, min_sep=1.2, seed=45),
    "hydrogen_rich": lambda: B.amorphous_carbon(300, h_fraction=0.5, density_g_cm3=1.2, min_sep=1.0, seed=46),
}


def _force(s, **kw):
    ctx = M.Context(potentials=M.POT_AIREBO, task_mode=1, **kw)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    try:
        return ctx.compute()
    except M.MdgError as err:
        return err.code
    finally:
        ctx.close()


@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("cap_cij", [0, 24])  # the default row, and one that some systems overflow
def test_group_build_equals_one_thread_build(name, cap_cij):
    s = SYSTEMS[name]()
    a, b = _force(s, cap_cij=cap_cij), _force(s, cap_cij=cap_cij, cap_bonds=40)
    if isinstance(a, int) or isinstance(b, int):
        assert a == b == -8  # MDG_ERR_CAPACITY from both
        return
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
