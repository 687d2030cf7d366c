"""Forwards of 129 to 192 heights in a batch: two banded parts in one 4-height body where
no other forward needs the 8-height body, else one part in that; heights past 256
never in more parts than the 8-height form's rest.  One launch per body."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib
from voxelproj_gb300.batch import FORWARD_DEFAULT, Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heights,launches", [
    ((180, 132, 192), 1), ((180, 64, 160), 1),   # the 4-height body alone
    ((180, 220), 1), ((132, 136, 236, 200), 1),  # the 8-height body alone
    ((180, 220, 64), 2), ((400, 448), 1), ((400, 160), 1), ((256, 140), 2),
    ((260,), 2),                                 # whole 256 and a rest of 4
])
def test_bodies(heights, launches):
    problems, checks = [], []
    for k, H in enumerate(heights):
        SY, SX, n, PX = 30 + k, 26, 21, 33
        ang = lin(n, -0.2, 3.3)
        x, y0 = seeded((SY, SX, H), 10 + k), seeded((n, PX, H), 20 + k)
        y = torch.tensor(y0, device="cuda")
        problems.append(("forward", torch.tensor(x, device="cuda"), y, torch.tensor(ang, device="cuda")))
        checks.append((y, y0, oracle.forward(x, ang, PX, 0)))
    batch = Batch(problems)
    before = _lib.LIB.vp_launch_count()
    batch.run()
    assert _lib.LIB.vp_launch_count() - before == launches
    for y, y0, want in checks:
        assert rel_err(y.cpu().numpy() - y0, want) <= tol.ref_vs_fp64(33)
    batch.close()


@pytest.mark.parametrize("SY,SX,n,PX", [(30, 26, 21, 33), (330, 320, 10, 300)])  # one slab, several
def test_parts_keep_the_sums_of_the_8_height_form(SY, SX, n, PX):
    a = torch.tensor(lin(n, -0.3, 3.4), device="cuda")
    problems, checks = [], []
    for H in (132, 140, 160, 192):
        x = torch.tensor(seeded((SY, SX, H), 97 + H), device="cuda")
        y = torch.tensor(seeded((n, PX, H), 98 + H), device="cuda")
        checks.append((x, y, y.clone()))
        problems.append(("forward", x, y, a))
    batch = Batch(problems)
    batch.run()
    assert not batch.error()
    _lib.LIB.vp_set_kernel_variant(0, FORWARD_DEFAULT)
    try:
        for x, y, want in checks:
            vp._CU.forward_z0(x, want, a)
            assert torch.equal(y, want)
    finally:
        _lib.LIB.vp_set_kernel_variant(0, 0)
    batch.close()
