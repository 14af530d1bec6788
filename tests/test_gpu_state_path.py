"""The way of a state between the caller and the device: positions outside the
box with their image counts, calls that follow mdg_set_state directly, and the
caller's arrays when the device reports an error.  States up to 4,096 atoms
pass through pinned memory in one copy, larger ones do not."""
import ctypes

import numpy as np
import pytest
import torch

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu

CELLS = [2, 8, 9]  # 64, 4,096 and 5,832 atoms


def _load(s, pot=M.POT_REBO, **kw):
    ctx = M.Context(potentials=pot, **kw)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    return ctx


def _moved(s, seed):
    """Positions up to 3 periods away on either side, with what wrapping them
    one rounded operation at a time gives."""
    rng = np.random.default_rng(seed)
    x = s["pos"] + rng.integers(-3, 4, size=s["pos"].shape) * s["box"]
    n = np.where((x < 0) | (x >= s["box"]), np.floor(x / s["box"]), 0.0)
    w = np.where(n != 0, x - n * s["box"], x)
    for _ in range(2):
        low, high = w < 0, w >= s["box"]
        w = np.where(low, w + s["box"], np.where(high, w - s["box"], w))
        n = n - low + high
    return x, w, n.astype(np.int32)


@pytest.mark.parametrize("cells", CELLS)
def test_positions_outside_the_box(cells):
    s = B.diamond(cells, temp_k=300.0, disp_sigma=0.05, seed=201)
    ctx = _load(s)
    p0, v0, m0 = ctx.get_state()
    x, w, n = _moved(s, 202)
    ctx.set_state(x)
    p, v, m = ctx.get_state()
    assert np.array_equal(p, w) and np.array_equal(v, v0) and np.array_equal(m, m0 + n)
    ctx.set_state(x, 2.0 * s["vel"])  # the periods add up
    p, v, m = ctx.get_state()
    assert np.array_equal(p, w) and np.array_equal(v, 2.0 * s["vel"]) and np.array_equal(m, m0 + 2 * n)


@pytest.mark.parametrize("cells", CELLS)
def test_calls_straight_after_set_state(cells):
    s = B.diamond(cells, temp_k=300.0, disp_sigma=0.05, seed=203)
    ctx = _load(s)
    p0 = ctx.get_state()[0]
    x, w, _ = _moved(s, 204)
    images = np.random.default_rng(205).integers(-9, 9, size=x.shape).astype(np.int32)
    ctx.set_state(x)
    ctx.set_images(images)
    assert np.array_equal(ctx.get_state()[2], images)
    ctx.set_state(x)
    ctx.set_state(p0, s["vel"])  # the second one's copy waits for the first's
    assert np.array_equal(ctx.get_state()[0], p0)
    other = torch.cuda.Stream()
    ctx.set_state(x)
    ctx.set_stream(other.cuda_stream)
    assert np.array_equal(ctx.get_state()[0], w)
    ctx.set_state(p0)
    ctx.set_stream(0)
    assert np.array_equal(ctx.get_state()[0], p0)
    t = B.ethane_liquid(30, seed=206)
    ctx.set_state(x)
    ctx.set_system(t["z"], t["pos"], t["vel"], t["box"], t["pbc"], t["fixed"])
    fresh = _load(t)
    assert np.array_equal(ctx.get_state()[0], fresh.get_state()[0])


@pytest.mark.parametrize("cells", CELLS)
def test_arrays_stay_when_the_device_reports_an_error(cells):
    s = B.diamond(cells, temp_k=300.0, seed=207)
    ctx = _load(s, task_mode=1, cap_bonds=1)
    ctx.run(1, 0.01, energies=False)  # the status is read by the next call that waits
    mark = [np.full((len(s["z"]), 3), 7.0), np.full((len(s["z"]), 3), 8.0), np.full((len(s["z"]), 3), 9, np.int32)]
    out = [a.copy() for a in mark]
    rc = M.lib().mdg_get_state(ctx.h, M._dp(out[0]), M._dp(out[1]), M._ip(out[2]))
    assert rc == -4  # MDG_ERR_BOND_OVERFLOW
    assert all(np.array_equal(a, b) for a, b in zip(out, mark))
    assert M.lib().mdg_get_state(ctx.h, M._dp(out[0]), None, M._ip(out[2])) == 0  # the error is reported once
    assert np.all(np.isfinite(out[0])) and not np.array_equal(out[0], mark[0])
    assert np.array_equal(out[1], mark[1])


def test_stream_destroyed_before_the_next_is_set():
    """A caller may destroy a stream as soon as its own calls on it are done;
    the state on its way there is waited for through the context's own event."""
    cu = ctypes.CDLL("libcuda.so.1")
    s = B.diamond(4, temp_k=300.0, disp_sigma=0.05, seed=208)
    ctx = _load(s)
    x, w, _ = _moved(s, 209)
    for _ in range(3):
        stream = ctypes.c_void_p()
        assert cu.cuStreamCreate(ctypes.byref(stream), 1) == 0  # CU_STREAM_NON_BLOCKING
        ctx.set_stream(stream.value)
        ctx.set_state(x)
        assert cu.cuStreamDestroy_v2(stream) == 0
        ctx.set_stream(0)
        assert np.array_equal(ctx.get_state()[0], w)
