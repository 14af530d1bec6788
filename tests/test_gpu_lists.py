"""Verlet pair sets against a k-d tree at the sizes where the list kernels
change: one block or several for the cells, a warp or a thread per atom, few or
many atoms a cell, too few cells for a grid, open and periodic axes, batches."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "one_atom_a_lane": lambda: B.c2h6_example(),
    "too_few_cells": lambda: B.ethane_liquid(29, seed=71),
    "odd": lambda: B.ethane_liquid(101, seed=72),
    "open_z": lambda: B.graphite_slab(3, 7, 5, temp_k=300.0, seed=73),
    "full_cells": lambda: B.diamond(8, disp_sigma=0.1, seed=74),
    "thread_build": lambda: B.diamond(13, disp_sigma=0.05, seed=75),   # 17,576 atoms
    "cells_in_kernels": lambda: B.diamond(21, disp_sigma=0.05, seed=76),  # 74,088 atoms
}
RANGE = (1.44 * 2.0, 1.44 * 5.5)


def _pairs(pos, s, r):
    span = np.where(s["pbc"] != 0, s["box"], 1e4)
    x = np.where(s["pbc"] != 0, np.mod(pos, span), pos - pos.min(axis=0) + 1.0)
    p = cKDTree(x, boxsize=span).query_pairs(r, output_type="ndarray")
    p.sort(axis=1)
    return p[np.lexsort((p[:, 1], p[:, 0]))].astype(np.int32)


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_lists_equal_a_kd_tree(name):
    s = SYSTEMS[name]()
    ctx = M.Context(potentials=M.POT_AIREBO)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    for shift in (0.0, 1.5):  # the first build, and a rebuild after every atom moved
        pos = s["pos"] + shift * np.random.default_rng(77).normal(size=3)
        if shift:
            ctx.set_state(pos)
        for l in (0, 1):
            # no pair of these systems lies within 1e-9 of a list range
            assert np.array_equal(ctx.nl_pairs(l), _pairs(pos, s, RANGE[l])), (name, shift, l)
    ctx.close()


def test_batched_lists_equal_single_ones():
    systems = [B.impact(81, n_target=900), B.ethane_liquid(30, seed=82), B.graphite_slab(2, 5, 3, seed=83)]
    ctx = M.Context(potentials=M.POT_AIREBO)
    ctx.set_batch(systems)
    for l in (0, 1):
        want, first = [], 0
        for s in systems:
            one = M.Context(potentials=M.POT_AIREBO)
            one.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
            want.append(one.nl_pairs(l) + first)
            first += len(s["z"])
        assert np.array_equal(ctx.nl_pairs(l), np.concatenate(want)), l
