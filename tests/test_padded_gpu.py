"""z_order 0 arrays whose rows are not whole, aligned float4: inputs are copied
with padded rows, outputs written by single heights."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded

pytestmark = pytest.mark.gpu


def _shifted(a, offset):
    """A CUDA copy of a whose data starts `offset` floats past an aligned address."""
    buf = torch.zeros(a.size + offset, device="cuda")
    t = buf[offset:].view(*a.shape)
    t.copy_(torch.from_numpy(a))
    return t


# (Hx, Hy): the first padded height count, remainders of 1 to 3 heights, of a
# 4-height part after the 8-height one, rows in float4 on one side only, more
# heights on one side; and aligned rows at an unaligned address (offset)
@pytest.mark.parametrize("Hx,Hy,offset", [(33, 33, 0), (34, 34, 0), (127, 127, 0), (129, 129, 0),
                                          (203, 203, 0), (257, 257, 0), (387, 387, 0),
                                          (512, 511, 0), (255, 256, 0), (40, 37, 0),
                                          (36, 36, 1), (256, 256, 2), (132, 132, 3)])
def test_rows_not_in_float4(Hx, Hy, offset):
    SY, SX, n, PX = 19, 26, 31, 29
    ang = lin(n, -0.2, 3.3)
    x, y = seeded((SY, SX, Hx), 51), seeded((n, PX, Hy), 52)
    H = min(Hx, Hy)
    a = torch.tensor(ang, device="cuda")
    yo, xo = _shifted(y, offset), _shifted(x, offset)
    vp._CU.forward_z0(_shifted(x, offset), yo, a)
    vp._CU.backward_z0(_shifted(y, offset), xo, a)
    Ax = oracle.forward(np.ascontiguousarray(x[..., :H]), ang, PX, 0)
    ATy = oracle.backward(np.ascontiguousarray(y[..., :H]), ang, SY, SX, 0)
    bound = tol.ref_vs_fp64(PX)
    assert rel_err(yo.cpu().numpy()[..., :H] - y[..., :H], Ax) <= bound
    assert rel_err(xo.cpu().numpy()[..., :H] - x[..., :H], ATy) <= bound
    # heights past the shorter array keep their values
    np.testing.assert_array_equal(yo.cpu().numpy()[..., H:], y[..., H:])
    np.testing.assert_array_equal(xo.cpu().numpy()[..., H:], x[..., H:])


def test_capture_without_copy():
    """Under stream capture the calls take no memory and run on the arrays
    themselves; the replayed result is the operator's."""
    SY, SX, H, n, PX = 19, 26, 45, 31, 29
    ang = lin(n)
    x, y = seeded((SY, SX, H), 53), seeded((n, PX, H), 54)
    a = torch.tensor(ang, device="cuda")
    xi, yi = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    yo, xo = torch.zeros_like(yi), torch.zeros_like(xi)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
        vp._CU.forward_z0(xi, yo, a)
        vp._CU.backward_z0(yi, xo, a)
    torch.cuda.current_stream().wait_stream(s)
    g.replay()
    bound = tol.ref_vs_fp64(PX)
    assert rel_err(yo.cpu().numpy(), oracle.forward(x, ang, PX, 0)) <= bound
    assert rel_err(xo.cpu().numpy(), oracle.backward(y, ang, SY, SX, 0)) <= bound
