"""Host arrays whose rows are not whole float4 (padded on arrival), few heights
(one step after another), and adjoints in one or several row slabs and chunks of
heights, in both output modes and with more heights on either side, against the
oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded

pytestmark = pytest.mark.gpu

N = 21


@pytest.mark.parametrize("z", [0, 2])
@pytest.mark.parametrize("Hx,Hy", [(1, 1), (1, 6), (3, 2), (4, 9), (5, 5), (7, 3), (9, 8), (8, 9),
                                   (31, 31), (33, 33), (45, 47), (130, 129), (203, 203), (257, 260), (300, 290)])
@pytest.mark.parametrize("SY,SX,PX", [(20, 26, 31), (150, 41, 90)])
def test_host_heights(SY, SX, PX, Hx, Hy, z):
    H = min(Hx, Hy)
    ang = lin(N, -0.3, 3.4)
    lay = (lambda v: v) if z == 0 else (lambda v: np.ascontiguousarray(np.moveaxis(v, 2, 0)))
    back = (lambda v: v) if z == 0 else (lambda v: np.moveaxis(v, 0, 2))
    x, y = seeded((SY, SX, Hx), 3), seeded((N, PX, Hy), 4)
    y_want = oracle.forward(np.ascontiguousarray(x[..., :H]), ang, PX, 0)
    x_want = oracle.backward(np.ascontiguousarray(y[..., :H]), ang, SY, SX, 0)
    bound = tol.ref_vs_fp64(max(SY, SX, PX))
    yo = lay(y).copy()
    vp.forward(lay(x), ang, yo, z_order=z)
    d = back(yo) - y
    assert rel_err(d[..., :H], y_want) <= bound and not d[..., H:].any()
    xo = lay(x).copy()
    vp.backward(lay(y), ang, xo, z_order=z)
    d = back(xo) - x
    assert rel_err(d[..., :H], x_want) <= bound and not d[..., H:].any()
    # a new output, of the other side's shape: past H zeros
    shape = (N, PX, Hy) if z == 0 else (Hy, N, PX)
    yn = back(vp.forward(lay(x), ang, shape, z_order=z))
    assert rel_err(yn[..., :H], y_want) <= bound and not yn[..., H:].any()
    shape = (SY, SX, Hx) if z == 0 else (Hx, SY, SX)
    xn = back(vp.backward(torch.from_numpy(lay(y)).pin_memory(), ang, shape, z_order=z).numpy())
    assert rel_err(xn[..., :H], x_want) <= bound and not xn[..., H:].any()


def test_several_slabs_with_padding():
    """Enough blocks for several row slabs, odd heights, pinned arrays: the device call's sums."""
    SY, SX, H, n, PX = 300, 260, 37, 40, 300
    ang = lin(n, -0.3, 3.4)
    x, y = seeded((SY, SX, H), 5), seeded((n, PX, H), 6)
    xd = torch.tensor(x, device="cuda")
    yd = torch.tensor(y, device="cuda")
    a = torch.tensor(ang, device="cuda")
    vp._CU.forward_z0(torch.tensor(x, device="cuda"), yd, a)
    vp._CU.backward_z0(torch.tensor(y, device="cuda"), xd, a)
    yh, xh = torch.from_numpy(y.copy()).pin_memory(), torch.from_numpy(x.copy()).pin_memory()
    vp.forward(torch.from_numpy(x).pin_memory(), ang, yh)
    vp.backward(torch.from_numpy(y).pin_memory(), ang, xh)
    # other groupings of the slabs' and angles' partial sums
    assert rel_err(yh.numpy(), yd.cpu().numpy()) <= 1e-6
    assert rel_err(xh.numpy(), xd.cpu().numpy()) <= 1e-6
