"""129 to 192 heights of the forward run as two banded parts where that takes less
than the 256-height form, more than 256 never: counted by launches (one slab each),
and the operator on both sides of the rule."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("SY,SX,H,n,PX,launches", [
    (40, 36, 132, 50, 40, 2), (40, 36, 192, 50, 40, 2),      # the GPU is not full
    (32, 32, 160, 300, 32, 1), (32, 32, 132, 300, 32, 1),    # small volume, enough blocks
    (64, 64, 160, 300, 64, 2), (64, 64, 164, 300, 64, 1),    # full: at most 160 heights
    (64, 64, 192, 264, 64, 2), (64, 64, 192, 268, 64, 1),    # a wave of 1064 blocks
    (64, 64, 400, 30, 64, 1), (64, 64, 448, 30, 64, 1),      # past 256 heights: no part of their own
    (64, 64, 300, 30, 64, 2),                                # a rest of at most 128: as ever
    (500, 410, 132, 5, 500, 7), (500, 410, 132, 6, 500, 5),  # few angles, large: 7 slabs, 4 + 1
])
def test_parts(SY, SX, H, n, PX, launches):
    ang = lin(n, -0.2, 3.3)
    x, y0 = seeded((SY, SX, H), 11), seeded((n, PX, H), 12)
    xt, a = torch.tensor(x, device="cuda"), torch.tensor(ang, device="cuda")
    y = torch.tensor(y0, device="cuda")
    before = _lib.LIB.vp_launch_count()
    vp._CU.forward_z0(xt, y, a)
    assert _lib.LIB.vp_launch_count() - before == launches
    assert rel_err(y.cpu().numpy() - y0, oracle.forward(x, ang, PX, 0)) <= tol.ref_vs_fp64(PX)
