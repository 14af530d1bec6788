"""Kernels that change with the size of a system.

Bond list and reverse slots run on eight lanes an atom up to a limit and on two
above it: a system on one side of the limit and a batch of its copies on the
other have the same forces, bit for bit (bond slots follow the atoms' numbers).

Connectivity: a group of lanes builds an atom's table unless its paths or bonds
do not fit; a bond capacity above 32 sends every atom to the one-thread build.
The paths of each system are counted here, so that both routes are known to be
taken, and tables that fit are compared bit for bit."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

BOND_R2 = {(6, 6): 2.0, (6, 1): 1.8, (1, 6): 1.8, (1, 1): 1.7}


def _force(s, pot=M.POT_AIREBO, **kw):
    ctx = M.Context(potentials=pot, task_mode=1, **kw)
    if isinstance(s, list):
        ctx.set_batch(s)
    else:
        ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    out = ctx.compute()
    ctx.close()
    return out


@pytest.mark.parametrize("build,copies", [
    (lambda: B.diamond(6, disp_sigma=0.08, seed=231), 39),                                                # 67,392 atoms
    (lambda: B.ethane_liquid(101, seed=232), 82),                                                         # 66,256
    (lambda: B.amorphous_carbon(500, h_fraction=0.4, density_g_cm3=1.2, min_sep=1.05, seed=233), 133),  # 66,500
])
@pytest.mark.parametrize("pot", [M.POT_REBO, M.POT_REBO | M.POT_ETORS, M.POT_BRENNER])
def test_a_system_and_a_batch_of_its_copies(build, copies, pot):
    s = build()
    e, et, g = _force(s, pot)
    f, ft, h = _force([s] * copies, pot)
    assert np.array_equal(h, np.tile(g, (copies, 1)))
    assert np.all(np.abs(ft - copies * et) <= 1e-12 * np.abs(ft))  # (summed in another order)


def _paths(s):
    """Bonds, paths of up to three bonds and their distinct ends, per atom."""
    z, n = s["z"], len(s["z"])
    span = np.where(s["pbc"] != 0, s["box"], 1e4)
    x = np.where(s["pbc"] != 0, np.mod(s["pos"], span), s["pos"] - s["pos"].min(axis=0) + 1.0)
    nb = [[] for _ in range(n)]
    for a, b in cKDTree(x, boxsize=span).query_pairs(2.0):
        d = x[a] - x[b]
        d -= np.where(s["pbc"] != 0, span * np.round(d / span), 0.0)
        if np.linalg.norm(d) < BOND_R2[z[a], z[b]]:
            nb[a].append(b)
            nb[b].append(a)
    count, ends = np.zeros(n, int), np.zeros(n, int)
    for i in range(n):
        seen = set()
        for k in nb[i]:
            two = [m for m in nb[k] if m != i]
            three = [t for m in two for t in nb[m] if t not in (i, k)]
            count[i] += 1 + len(two) + len(three)
            seen.update([k], two, three)
        ends[i] = len(seen)
    return np.array([len(v) for v in nb]), count, ends


SYSTEMS = {  # name: (system, some atom's bonds or paths do not fit a group, some atom has more than 23 ends)
    "molecule": (lambda: B.c2h6_example(), False, False),
    "graphite": (lambda: B.graphite_slab(2, 5, 3, temp_k=2000.0, seed=42), False, False),
    "diamond": (lambda: B.diamond(4, disp_sigma=0.12, seed=43), False, True),
    "dense": (lambda: B.amorphous_carbon(400, density_g_cm3=2.6, min_sep=1.2, seed=45), True, True),
    "hydrogen_rich": (lambda: B.amorphous_carbon(300, h_fraction=0.5, density_g_cm3=1.2, min_sep=1.0, seed=46),
                      False, True),
}
ROOM = dict(cap_special=512, special_avg=512, cap_lj_list=1024, bond_rec_avg=1024)  # for all but the table


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_tables_that_fit_are_the_same(name):
    build, beyond, _ = SYSTEMS[name]
    s = build()
    bonds, paths, ends = _paths(s)
    assert (bonds.max() > 8 and paths.max() > 128) == beyond and ends.max() < 127
    assert bonds.min() <= 8 and paths.min() <= 128  # the groups are taken too
    a, b = _force(s, **ROOM), _force(s, cap_bonds=40, **ROOM)
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_tables_that_do_not_fit_are_reported(name):
    """A table of 24 places holds 23 ends and the atom itself."""
    build, _, over = SYSTEMS[name]
    s = build()
    assert (_paths(s)[2].max() > 23) == over
    for kw in (ROOM, dict(cap_bonds=40, **ROOM)):
        if over:
            with pytest.raises(M.MdgError) as err:
                _force(s, cap_cij=24, **kw)
            assert err.value.code == -8
        else:
            a, b = _force(s, cap_cij=24, **kw), _force(s, **kw)
            assert a[0] == b[0] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("edge", [40.0, 90.0, 100.0])  # 2,197, 29,791 and 39,304 cells: the cluster, the cluster, four kernels
def test_lists_of_a_gas_equal_a_kd_tree(edge):
    m = B.c2h6_example()
    place = (np.stack(np.meshgrid(*3 * [np.arange(3)], indexing="ij"), -1).reshape(-1, 1, 3) + 0.5) * edge / 3
    pos = (place + m["pos"] - m["pos"].mean(axis=0)).reshape(-1, 3)
    pos += np.random.default_rng(234).normal(scale=0.02, size=pos.shape)
    ctx = M.Context(potentials=M.POT_REBO)
    ctx.set_system(np.tile(m["z"], 27), pos, None, 3 * [edge])
    for shift in (0.0, 0.37 * edge):  # the second time through the borders
        x = np.mod(pos + shift, edge)
        ctx.set_state(x)
        want = cKDTree(x, boxsize=edge).query_pairs(1.44 * 2.0, output_type="ndarray")
        want.sort(axis=1)
        # (no pair lies within 1e-9 of the range)
        assert np.array_equal(ctx.nl_pairs(0), want[np.lexsort((want[:, 1], want[:, 0]))])
