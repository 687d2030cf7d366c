"""Host arrays of odd heights: calls pad their rows on arrival (one more launch per
piece) only from the angle counts on where that pays."""

from __future__ import annotations

import numpy as np
import pytest

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


def _launches(S, H, n, check, forward=True):
    ang = lin(n, -0.2, 3.3)
    x = seeded((S, S, H), 5)
    before = _lib.LIB.vp_launch_count()
    if not forward:
        y = seeded((n, S, H), 6)
        before = _lib.LIB.vp_launch_count()
        z = vp.backward(y, ang, None)
        count = _lib.LIB.vp_launch_count() - before
        assert rel_err(z, oracle.backward(y, ang, S, S, 0)) <= tol.ref_vs_fp64(S)
        return count
    y = vp.forward(x, ang, None)
    count = _lib.LIB.vp_launch_count() - before
    if check:
        assert rel_err(y, oracle.forward(x, ang, S, 0)) <= tol.ref_vs_fp64(S)
    return count


@pytest.mark.parametrize("S,H,line", [(192, 203, 30), (104, 257, 100), (64, 203, 240)])
def test_padding_starts_where_it_pays(S, H, line):
    below = [_launches(S, H, n, check=S == 64) for n in (line // 2, line - 1)]
    assert below[0] == below[1] < _launches(S, H, line, check=S == 64)


@pytest.mark.parametrize("S,H,line", [(64, 9, 120), (192, 15, 90), (128, 33, 45), (128, 99, 30), (64, 33, 90), (96, 99, 60), (30, 99, 120), (30, 203, 200)])
def test_adjoint_padding_starts_where_it_pays(S, H, line):
    below = [_launches(S, H, n, True, forward=False) for n in (line // 2, line - 1)]
    assert below[0] == below[1] < _launches(S, H, line, True, forward=False)
