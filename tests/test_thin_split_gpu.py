"""The adjoint of few heights with the angles split over a block's four warps: equal
shares at any number of angles, and the kernels for fewer than 8 of them."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded, x_shape, y_shape

pytestmark = pytest.mark.gpu


def _time(H, S, n):
    """Shortest of several backward calls on a (H, S, S) volume, in ms."""
    a = torch.tensor(lin(n), device="cuda")
    y, x = torch.randn(H, n, S, device="cuda"), torch.zeros(H, S, S, device="cuda")
    best = float("inf")
    for _ in range(6):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        for _ in range(20):
            vp._CU.backward_z2(y, x, a)
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best


@pytest.mark.parametrize("H,S", [(8, 256), (2, 512)])
def test_few_angles_are_shared(H, S):
    """32 angles are a quarter of 128: with all of them on one of the four warps they took
    about as long."""
    assert _time(H, S, 32) <= 0.55 * _time(H, S, 128)


@pytest.mark.parametrize("z", [0, 2])
@pytest.mark.parametrize("H", [1, 2, 3, 5, 7, 12])
@pytest.mark.parametrize("n", [1, 3, 7, 8, 9, 31, 33, 127, 128, 129, 130, 161, 257])
def test_angle_counts(n, H, z):
    SY, SX, PX = (33, 29, 41) if n % 2 else (25, 24, 30)
    ang = lin(n, -0.3, 6.1)
    y, x0 = seeded(y_shape(z, n, PX, H), 31), seeded(x_shape(z, SY, SX, H), 32)
    x = torch.tensor(x0, device="cuda")
    (vp._CU.backward_z0 if z == 0 else vp._CU.backward_z2)(
        torch.tensor(y, device="cuda"), x, torch.tensor(ang, device="cuda"))
    want = oracle.backward(y, ang, SY, SX, z)
    assert rel_err(x.cpu().numpy() - x0, want) <= tol.ref_vs_fp64(PX)
