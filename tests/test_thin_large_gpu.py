"""The adjoint of few heights in volumes large enough that a block's warps take
neighbouring rows (no split of the angles), and with four voxels per lane, split and
not: last rows and columns partial, both layouts, both output modes, both trig modes."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded, x_shape, y_shape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trig", ["reference", "precise"])
@pytest.mark.parametrize("SY,SX,H,z", [
    (390, 380, 13, 2), (390, 380, 16, 2),                               # one voxel, unsplit
    (515, 260, 1, 0), (515, 260, 2, 0), (515, 260, 3, 0),               # four voxels, split
    (515, 260, 1, 2), (515, 260, 2, 2), (515, 260, 4, 2),
    (1030, 517, 1, 0), (1030, 517, 2, 0), (1030, 517, 3, 0),            # four voxels, unsplit
    (1030, 517, 1, 2), (1030, 517, 2, 2), (1030, 517, 3, 2), (1030, 517, 4, 2),
    (1030, 517, 7, 0), (1030, 517, 5, 2),                               # one voxel, unsplit
])
def test_large_volumes(SY, SX, H, z, trig):
    n, PX = 11, SY - 20
    ang = lin(n, -0.3, 6.1)
    y, x0 = seeded(y_shape(z, n, PX, H), 71), seeded(x_shape(z, SY, SX, H), 72)
    yt, a = torch.tensor(y, device="cuda"), torch.tensor(ang, device="cuda")
    vp.set_trig_mode(trig)
    try:
        added = torch.tensor(x0, device="cuda")
        (vp._CU.backward_z0 if z == 0 else vp._CU.backward_z2)(yt, added, a)
        stored = torch.full_like(added, float("nan"))
        vp._CU.project_store(False, z, yt, stored, a)
    finally:
        vp.set_trig_mode("reference")
    want = oracle.backward(y, ang, SY, SX, z)
    bound = tol.precise_vs_fp64(SY) if trig == "precise" else tol.ref_vs_fp64(SY)
    assert rel_err(added.cpu().numpy() - x0, want) <= bound
    assert rel_err(stored.cpu().numpy(), want) <= bound
