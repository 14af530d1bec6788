"""LJ pairs outside the bond-order window (r > 2^(1/6) sigma), which run from
1/r^2 with a root only inside the cutoff's cosine window.

Isolated pairs against f(r) 4 eps [(s/r)^12 - (s/r)^6] in numpy, in terms of
the sum of the two powers' magnitudes.  FP64: some ten roundings, and 0.5 - 0.5
of the window's cosine is rounded at 1e-16: 1e-14 leaves a margin of ten.  Mixed:
the window's argument takes r in float, half a last place of which is 2.4e-7 A
below 8 A and 4.8e-7 above, so pi / 0.5 A times that for the argument, half of
it for f, and the window's derivative pi / 1 A times that again: 2e-6 of the
pair's own scale and 1e-5 of the window's.

A liquid and a crystal against the general form that the derivative pass keeps."""
import numpy as np
import pytest

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

SIGMA = {(6, 6): 3.40, (1, 1): 2.65, (1, 6): 0.5 * (3.40 + 2.65)}
EPS = {(6, 6): 0.00284, (1, 1): 0.00150, (1, 6): np.sqrt(0.00284 * 0.00150)}
R1 = {(6, 6): 5.0, (1, 1): 4.0, (1, 6): 4.5}


def _window(t, cut_mode):
    return (3.0 * SIGMA[t] - 0.5, 3.0 * SIGMA[t]) if cut_mode else (R1[t], R1[t] + 0.5)


def _pairs(cut_mode):
    out = []
    for t in sorted(SIGMA):
        a, b = _window(t, cut_mode)
        lo = 2.0 ** (1.0 / 6.0) * SIGMA[t]
        r = np.concatenate([np.linspace(lo + 1e-6, a, 14), np.linspace(a, b, 15), a + np.array([-1e-9, 1e-9]),
                            b + np.array([-1e-9, 1e-9, 0.1])])
        out += [(t, x, k) for k, x in enumerate(r)]
    return out


@pytest.mark.parametrize("cut_mode", [0, 1])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_FP32_MIXED])
def test_isolated_pairs(cut_mode, precision):
    rng = np.random.default_rng(221)
    systems, want_e, want_g, tol_e, tol_g = [], [], [], [], []
    for t, r, k in _pairs(cut_mode):
        u = rng.normal(size=3)
        x = np.array([[8.0, 9.0, 10.0], [8.0, 9.0, 10.0] + r * u / np.linalg.norm(u)])
        z = np.array(t if k % 2 else t[::-1], np.int32)  # either species first
        systems.append(dict(z=z, pos=x, vel=np.zeros((2, 3)), box=np.zeros(3), pbc=np.zeros(3, np.int32),
                            fixed=np.zeros(2, np.uint8)))
        d = x[0] - x[1]
        r = np.sqrt((d * d).sum())
        a, b = _window(t, cut_mode)
        s6 = (SIGMA[t] / r) ** 6
        v = 4.0 * EPS[t] * (s6 * s6 - s6)
        dv = 4.0 * EPS[t] * (6.0 * s6 - 12.0 * s6 * s6) / r
        f, df = 1.0, 0.0
        if r >= a:
            p = np.pi * (r - a) / (b - a)
            f, df = (0.5 + 0.5 * np.cos(p), -0.5 * np.pi / (b - a) * np.sin(p)) if r <= b else (0.0, 0.0)
        want_e.append(f * v)
        g = (f * dv + df * v) / r * d
        want_g += [g, -g]
        scale = 4.0 * EPS[t] * (s6 * s6 + s6)
        inside = 4.0 * EPS[t] * (12.0 * s6 * s6 + 6.0 * s6) / r
        if precision == M.PREC_FP64:
            tol_e.append(1e-14 * scale)
            tol_g += 2 * [1e-14 * (inside + np.pi * scale)]
        else:
            tol_e.append(2e-6 * scale)
            tol_g += 2 * [2e-6 * inside + 1e-5 * scale]
    ctx = M.Context(potentials=M.POT_AIREBO, precision=precision, lj_cut_mode=cut_mode)
    ctx.set_batch(systems)
    e = ctx.batch_energies()
    _, _, g = ctx.compute()
    assert np.all(e[:, [0, 2, 3]] == 0.0)
    assert np.all(np.abs(e[:, 1] - np.array(want_e)) <= tol_e)
    assert np.all(np.linalg.norm(g - np.array(want_g), axis=1) <= tol_g)


@pytest.mark.parametrize("build,cut_mode", [
    (lambda: B.ethane_liquid(101, seed=222), 0), (lambda: B.ethane_liquid(101, seed=222), 1),
    (lambda: B.graphite_slab(3, 7, 5, temp_k=300.0, seed=223), 0)])
def test_force_call_equals_the_derivative_pass(build, cut_mode):
    """The gradient of the derivative pass goes through the general form of
    every far pair.  (Systems without bonds in the cutoffs' windows: there the
    force call gives the reference's force, not the energy's exact gradient.)
    Both add the same terms in other orders; a force of the bond-order tables
    keeps about 2e-10 of such rounding."""
    s = build()
    ctx = M.Context(potentials=M.POT_AIREBO, lj_cut_mode=cut_mode, cap_lj_list=2048)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    _, _, g = ctx.compute()
    d = ctx.force_product(np.zeros_like(s["pos"]))["grad"]
    assert np.linalg.norm(g - d) <= 1e-9 * np.linalg.norm(d)
