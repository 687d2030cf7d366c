"""z_order 2 forwards of few heights: an infinite voxel reaches the bins that it has a
weight in and no others, with scratch (transposed, banded) and without."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests.common import lin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("trig", ["reference", "precise"])
@pytest.mark.parametrize("H", [1, 4, 5, 8, 13, 16, 17, 31])
@pytest.mark.parametrize("SY,SX,PX", [(30, 26, 29), (70, 100, 90)])
def test_infinite_voxel(SY, SX, PX, H, trig, host):
    n = 41
    ang = lin(n, 0.05, 3.1)
    voxel = (H // 2, SY // 3, SX // 2)
    unit = np.zeros((1, SY, SX), np.float32)
    unit[0, voxel[1], voxel[2]] = 1.0
    # weights nearby in angle: what rounding of the angle's constants could reach
    w = np.stack([oracle.forward(unit, ang + np.float32(d), PX, 2)[0] for d in (-1e-4, 0.0, 1e-4)])
    x = np.random.default_rng(H).standard_normal((H, SY, SX)).astype(np.float32)
    x[voxel] = np.inf
    vp.set_trig_mode(trig)
    try:
        if host:
            y = vp.forward(x, ang, None if PX == max(SY, SX) else (H, n, PX), z_order=2)
        else:
            y = vp.forward(torch.tensor(x, device="cuda"), ang, (H, n, PX), z_order=2).cpu().numpy()
    finally:
        vp.set_trig_mode("reference")
    finite = np.isfinite(y)
    assert finite[np.arange(H) != voxel[0]].all()
    assert finite[voxel[0]][w.max(axis=0) == 0].all()
    assert not finite[voxel[0]][w.min(axis=0) > 1e-3].any()
