"""The energy rows of captured steps: runs with and without energies in turn,
logs that grow, and batch runs beside runs in one context, against one run over
all steps.  Each step is the same launches with the same arguments, so the
values are the same bit for bit; a batch's total is summed in another order
than its systems (1e-12)."""
import numpy as np
import pytest

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pot", [M.POT_REBO, M.POT_AIREBO, M.POT_BRENNER])
def test_rows_of_runs_in_pieces(pot):
    s = B.ethane_liquid(60, seed=211, min_dist=1.6, jitter=0.4)

    def load():
        ctx = M.Context(potentials=pot, task_mode=2)
        ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
        return ctx

    pieces = [(3, True), (2, False), (1, True), (70, True), (0, True), (4, False), (20, True)]
    a, b = load(), load()
    ep, et = a.run(sum(k for k, _ in pieces), 0.25)
    at = 0
    for k, energies in pieces:
        out = b.run(k, 0.25, energies=energies)
        if energies:
            assert np.array_equal(out[0], ep[at:at + k]) and np.array_equal(out[1], et[at:at + k]), (at, k)
        at += k
    for x, y in zip(a.get_state(), b.get_state()):
        assert np.array_equal(x, y)


def test_rows_of_batch_runs_beside_runs():
    systems = [B.ethane_liquid(30, seed=212), B.diamond(4, temp_k=300.0, seed=213), B.graphite_slab(2, 5, 3, seed=214)]

    def load():
        ctx = M.Context(potentials=M.POT_AIREBO, task_mode=2)
        ctx.set_batch(systems)
        return ctx

    pieces = [(2, "batch"), (3, "run"), (9, "batch"), (4, "none"), (30, "run"), (6, "batch"), (1, "run")]
    a, b = load(), load()
    ep, et = a.batch_run(sum(k for k, _ in pieces), 0.25)
    at = 0
    for k, kind in pieces:
        if kind == "batch":
            p, t = b.batch_run(k, 0.25)
            assert np.array_equal(p, ep[at:at + k]) and np.array_equal(t, et[at:at + k]), (at, k)
        elif kind == "run":
            p, t = b.run(k, 0.25)
            assert np.allclose(p, ep[at:at + k].sum(1), rtol=1e-12, atol=0)
            assert np.allclose(t, et[at:at + k].sum(1), rtol=1e-12, atol=0)
        else:
            b.run(k, 0.25, energies=False)
        at += k
    for x, y in zip(a.get_state(), b.get_state()):
        assert np.array_equal(x, y)
