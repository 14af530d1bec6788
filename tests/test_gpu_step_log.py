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


@pytest.mark.parametrize("energies", [True, False])
def test_a_final_time_set_between_runs(energies):
    """Systems of adaptive dt stop at the final time that stands when a run
    begins, also where an earlier one was in force when the step was captured."""
    systems = [B.diamond(4, temp_k=t, disp_sigma=0.02, seed=215 + k) for k, t in enumerate((300.0, 1200.0))]

    def load(final):
        ctx = M.Context(potentials=M.POT_REBO, task_mode=1)
        ctx.set_batch(systems)
        ctx.set_adaptive_dt(True, 1.0, 0.5)
        ctx.set_time_final(final)
        ctx.set_stop_at_time_final(True)
        return ctx

    def run(ctx, steps):
        if energies:
            ctx.batch_run(steps, 0.5)
        else:
            ctx.run(steps, 0.5, energies=False)

    a, b = load(10.0), load(2.0)
    run(b, 8)  # 2 fs at 0.5 fs a step or less: both systems end on the way
    assert (b.get_time()[0] >= 2.0).all() and (b.get_time()[0] <= 2.5).all()
    b.set_time_final(10.0)
    run(b, 40)
    run(a, 48)
    assert (b.get_time()[0] >= 10.0).all() and (b.get_time()[0] <= 10.5).all()
    assert np.array_equal(a.get_time()[0], b.get_time()[0])
    # (a stopped system's forces are taken again at its wrapped positions: equal to rounding)
    for x, y in zip(a.get_state(), b.get_state()):
        assert np.allclose(x, y, rtol=0, atol=1e-9)
