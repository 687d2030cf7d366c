"""Host arrays of odd heights past 192: the forward pads its rows on arrival (one more
launch per piece) only from the angle counts on where that pays."""

from __future__ import annotations

import numpy as np
import pytest

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


def _launches(S, H, n, check):
    ang = lin(n, -0.2, 3.3)
    x = seeded((S, S, H), 5)
    before = _lib.LIB.vp_launch_count()
    y = vp.forward(x, ang, None)
    count = _lib.LIB.vp_launch_count() - before
    if check:
        assert rel_err(y, oracle.forward(x, ang, S, 0)) <= tol.ref_vs_fp64(S)
    return count


@pytest.mark.parametrize("S,H,line", [(192, 203, 30), (104, 257, 100), (64, 203, 240)])
def test_padding_starts_where_it_pays(S, H, line):
    below = [_launches(S, H, n, check=S == 64) for n in (line // 2, line - 1)]
    assert below[0] == below[1] < _launches(S, H, line, check=S == 64)
