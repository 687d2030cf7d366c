"""Row slabs of the z_order 0 adjoint with host arrays: above 128 heights with fewer than
256 angles half as many blocks make one, so there are more (counted by launches)."""

from __future__ import annotations

import pytest

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


def _launches(S, H, n):
    ang = lin(n, -0.2, 3.3)
    y = seeded((n, S, H), 5)
    before = _lib.LIB.vp_launch_count()
    x = vp.backward(y, ang, None)
    count = _lib.LIB.vp_launch_count() - before
    if n < 100:
        assert rel_err(x, oracle.backward(y, ang, S, S, 0)) <= tol.ref_vs_fp64(S)
    return count


@pytest.mark.parametrize("S,H,more", [(160, 256, True), (160, 160, True), (160, 128, False)])
def test_slabs(S, H, more):
    few, many = _launches(S, H, 30), _launches(S, H, 256)
    assert _launches(S, H, 255) == few
    assert few > many if more else few == many
