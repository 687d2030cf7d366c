"""The z_order 0 adjoint with host arrays sums the first sixth of the angles and the rest
apart, whatever the sinogram's size: the device calls on the two groups bit for bit."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests.common import lin, seeded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("SY,SX,H,n,PX", [(29, 50, 152, 50, 66), (32, 32, 32, 128, 32),
                                          (64, 64, 64, 100, 64), (40, 36, 12, 7, 40),
                                          (96, 80, 128, 120, 96)])  # 5.9 MB: in two pieces
def test_two_groups_of_angles(SY, SX, H, n, PX):
    ang = lin(n, -0.2, 3.2)
    y = seeded((n, PX, H), 3)
    got = vp.backward(torch.from_numpy(y).pin_memory(), ang, (SY, SX, H))
    k = n // 6 if n >= 8 else 0
    yt, a = torch.tensor(y, device="cuda"), torch.tensor(ang, device="cuda")
    x = torch.zeros(SY, SX, H, device="cuda")
    for lo, hi in ((0, k), (k, n)):
        if hi > lo:
            vp._CU.backward_z0(yt[lo:hi].contiguous(), x, a[lo:hi].contiguous())
    assert torch.equal(got, x.cpu())
