"""What the derivative pass holds on the GPU."""
import pytest
import torch

import mdtk_b200 as M
from mdtk_b200 import builders as B

pytestmark = pytest.mark.gpu


def _held(s, **kw):
    """Bytes a first pass takes."""
    ctx = M.Context(potentials=M.POT_AIREBO, task_mode=1, **kw)
    ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
    ctx.compute()
    ctx.sync()
    before = torch.cuda.mem_get_info()[0]
    ctx.force_product(s["vel"])
    after = torch.cuda.mem_get_info()[0]
    ctx.close()
    return before - after


def test_bond_records_share_the_special_pairs_memory():
    """Records of 8,000 atoms at twice the default capacity are 131 MB; the
    special pairs' are 172 MB, and no larger for them."""
    s = B.diamond(10, temp_k=600.0, disp_sigma=0.05, seed=251)
    _held(s)  # (the kernels' own memory)
    a, b = _held(s), _held(s, bond_rec_avg=512)
    assert abs(b - a) <= 8 << 20  # (allocations come in pieces of 2 MB)


@pytest.mark.parametrize("rec", [256, 512, 1024])
def test_gradients_do_not_depend_on_where_the_records_lie(rec):
    s = B.diamond(5, temp_k=600.0, disp_sigma=0.05, seed=252)
    out = []
    for kw in ({}, dict(bond_rec_avg=rec)):  # 1,024: records of their own
        ctx = M.Context(potentials=M.POT_AIREBO, task_mode=1, **kw)
        ctx.set_system(s["z"], s["pos"], s["vel"], s["box"], s["pbc"], s["fixed"])
        out.append(ctx.force_product(s["vel"]))
        ctx.close()
    for k in out[0]:
        assert (out[0][k] == out[1][k]).all(), k
