"""z_order 0 rows that are not whole float4 are copied with padded rows only where
the copy pays: one launch (the scalar kernel) below the line, the copy and the
float4 kernels above it; the operator on both sides."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


# (operator, SY, SX, H, angles, PX, launches): the adjoint's float4 form is the
# copy and a launch per angle class (and the same for a rest past 256 heights),
# the forward's the copy and one launch
@pytest.mark.parametrize("op,SY,SX,H,n,PX,launches", [
    ("backward", 64, 64, 9, 59, 64, 1), ("backward", 64, 64, 9, 60, 64, 3),
    ("backward", 24, 24, 203, 119, 24, 1), ("backward", 24, 24, 203, 120, 24, 3),
    ("backward", 64, 64, 99, 60, 257, 1), ("backward", 130, 128, 33, 15, 130, 1),
    ("backward", 130, 128, 33, 16, 130, 3), ("backward", 130, 128, 31, 59, 130, 1),
    ("backward", 260, 256, 9, 29, 260, 1), ("backward", 260, 256, 9, 30, 260, 3),
    ("backward", 30, 26, 257, 4, 30, 1), ("backward", 24, 24, 99, 59, 24, 1),
    ("backward", 24, 24, 99, 60, 24, 3), ("backward", 96, 96, 203, 15, 96, 1),
    ("backward", 96, 96, 203, 16, 96, 3), ("backward", 45, 45, 401, 59, 45, 1),
    ("backward", 48, 48, 401, 60, 48, 3),
    ("forward", 24, 24, 131, 3, 24, 1), ("forward", 48, 48, 99, 1, 48, 2),
    ("forward", 24, 24, 203, 239, 24, 1), ("forward", 24, 24, 203, 240, 24, 2),
    ("forward", 70, 64, 203, 59, 70, 1), ("forward", 64, 64, 255, 60, 64, 2),
    ("forward", 130, 128, 203, 29, 130, 1), ("forward", 36, 33, 203, 119, 36, 1),
    ("forward", 36, 33, 203, 120, 36, 2), ("forward", 20, 100, 203, 120, 100, 1),
    ("forward", 96, 96, 255, 59, 96, 1), ("forward", 40, 240, 255, 59, 240, 1),
])
def test_copy_where_it_pays(op, SY, SX, H, n, PX, launches):
    ang = lin(n, -0.2, 3.3)
    a = torch.tensor(ang, device="cuda")
    x, y = seeded((SY, SX, H), 21), seeded((n, PX, H), 22)
    forward = op == "forward"
    src, dst = (x, y) if forward else (y, x)
    out = torch.tensor(dst, device="cuda")
    inp = torch.tensor(src, device="cuda")
    before = _lib.LIB.vp_launch_count()
    (vp._CU.forward_z0 if forward else vp._CU.backward_z0)(inp, out, a)
    assert _lib.LIB.vp_launch_count() - before == launches
    want = oracle.forward(x, ang, PX, 0) if forward else oracle.backward(y, ang, SY, SX, 0)
    assert rel_err(out.cpu().numpy() - dst, want) <= tol.ref_vs_fp64(max(SY, SX, PX))


# (Hx, Hy, floats past an aligned address): remainders of 1 to 3 heights, of a 4-height
# part after the 8-height one, float4 rows on one side only, unaligned rows
@pytest.mark.parametrize("Hx,Hy,offset", [(9, 9, 0), (33, 33, 0), (34, 34, 0), (127, 127, 0), (203, 203, 0),
                                          (257, 257, 0), (387, 387, 0), (512, 511, 0), (255, 256, 0),
                                          (40, 37, 0), (36, 36, 1), (256, 256, 2), (132, 132, 3)])
def test_padded_rows(Hx, Hy, offset):
    SY, SX, n, PX = 70, 64, 61, 67
    ang = lin(n, -0.2, 3.3)
    x, y = seeded((SY, SX, Hx), 51), seeded((n, PX, Hy), 52)
    H = min(Hx, Hy)
    a = torch.tensor(ang, device="cuda")

    def shifted(v):
        t = torch.zeros(v.size + offset, device="cuda")[offset:].view(*v.shape)
        return t.copy_(torch.from_numpy(v))

    yo, xo = shifted(y), shifted(x)
    before = _lib.LIB.vp_launch_count()
    vp._CU.forward_z0(shifted(x), yo, a)
    vp._CU.backward_z0(shifted(y), xo, a)
    copies = (Hx % 4 != 0 or offset > 0) + (Hy % 4 != 0 or offset > 0)
    assert _lib.LIB.vp_launch_count() - before >= 3 + copies
    Ax = oracle.forward(np.ascontiguousarray(x[..., :H]), ang, PX, 0)
    ATy = oracle.backward(np.ascontiguousarray(y[..., :H]), ang, SY, SX, 0)
    bound = tol.ref_vs_fp64(SY)
    assert rel_err(yo.cpu().numpy()[..., :H] - y[..., :H], Ax) <= bound
    assert rel_err(xo.cpu().numpy()[..., :H] - x[..., :H], ATy) <= bound
    np.testing.assert_array_equal(yo.cpu().numpy()[..., H:], y[..., H:])
    np.testing.assert_array_equal(xo.cpu().numpy()[..., H:], x[..., H:])
