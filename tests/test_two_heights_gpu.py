"""The run adjoint with 2 heights per lane (at most 64 heights, or such a rest): the
sums of the form with 4 heights per lane bit for bit, whole and partial last lanes,
outputs by float2 and by single heights, single and several row slabs."""

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


@pytest.mark.parametrize("H", [4, 8, 12, 28, 32, 36, 60, 64, 68, 260, 300, 320])
@pytest.mark.parametrize("SY,SX,PX", [(33, 18, 40), (70, 65, 52)])
def test_equals_four_heights_per_lane(SY, SX, PX, H):
    a = torch.tensor(lin(37, -0.3, 6.4), device="cuda")
    y = torch.tensor(seeded((37, PX, H), 1), device="cuda")
    x = torch.tensor(seeded((SY, SX, H), 2), device="cuda")
    want = x.clone()
    vp._CU.backward_z0(y, x, a)
    _lib.LIB.vp_set_kernel_variant(1, 7)
    try:
        vp._CU.backward_z0(y, want, a)
    finally:
        _lib.LIB.vp_set_kernel_variant(1, 0)
    assert torch.equal(x, want)


@pytest.mark.parametrize("Hx,Hy", [(9, 9), (19, 20), (20, 19), (31, 33), (63, 62), (65, 65), (5, 4),
                                   (4, 6), (290, 291)])
def test_odd_heights_match_oracle(Hx, Hy):
    SY, SX, n, PX = 45, 38, 31, 57
    H = min(Hx, Hy)
    ang = lin(n, -0.3, 6.4)
    y, x0 = seeded((n, PX, Hy), 3), seeded((SY, SX, Hx), 4)
    x = torch.tensor(x0, device="cuda")
    vp._CU.backward_z0(torch.tensor(y, device="cuda"), x, torch.tensor(ang, device="cuda"))
    d = x.cpu().numpy() - x0
    want = oracle.backward(np.ascontiguousarray(y[..., :H]), ang, SY, SX, 0)
    assert rel_err(d[..., :H], want) <= tol.ref_vs_fp64(PX) and not d[..., H:].any()
