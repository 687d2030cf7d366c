"""The z_order 2 adjoint with host arrays goes by equal halves where few angles leave
the copies in charge, and by whole 128- and 256-height chunks where the kernels take
the time: up to 128 heights told apart by launches, the operator either way."""

from __future__ import annotations

import numpy as np
import pytest

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


def _launches(H, S, n, check):
    ang = lin(n, -0.2, 3.3)
    y, x0 = seeded((H, n, S), 5), seeded((H, S, S), 6)
    x = x0.copy()
    before = _lib.LIB.vp_launch_count()
    vp.backward(y, ang, x, z_order=2)
    count = _lib.LIB.vp_launch_count() - before
    if check:
        assert rel_err(x - x0, oracle.backward(y, ang, S, S, 2)) <= tol.ref_vs_fp64(S)
    return count


def test_halves_with_few_angles():
    assert _launches(66, 300, 74, check=True) != _launches(66, 300, 75, check=False)


@pytest.mark.parametrize("H,S,n", [(66, 299, 20), (257, 199, 20), (140, 200, 20), (520, 60, 20)])
def test_same_chunks_where_the_rule_does_not_reach(H, S, n):
    assert _launches(H, S, n, check=S < 100) == _launches(H, S, 110, check=False)


@pytest.mark.parametrize("H", [257, 300, 511])  # two unequal, two equal, two nearly equal chunks
def test_two_chunks(H):
    _launches(H, 200, 11, check=True)
