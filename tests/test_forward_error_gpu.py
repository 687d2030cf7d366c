"""The default forward's error against 64 bits is no larger than that of the candidate
lists, whose sums it regroups: an accumulator that runs over more lines has more."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests.common import lin
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


# variant 13: a run's lines on two warps, 16: one warp; both in slabs
@pytest.mark.parametrize("SY,SX,H,n,PX,lists", [
    (500, 512, 32, 50, 512, 16), (500, 512, 8, 50, 512, 16), (64, 64, 100, 400, 64, 13),
    (116, 116, 80, 160, 116, 13), (256, 256, 160, 30, 256, 16), (24, 24, 100, 300, 24, 13),
])
def test_error_no_larger_than_the_lists(SY, SX, H, n, PX, lists):
    ang = lin(n, 0.0, 3.1)
    rng = np.random.default_rng(5)
    # densities around one: rounding errors of a long sum do not cancel
    x = (1.0 + 0.3 * rng.standard_normal((SY, SX, H))).astype(np.float32)
    want = oracle.forward(x, ang, PX, 0)
    xt, a = torch.tensor(x, device="cuda"), torch.tensor(ang, device="cuda")
    err = {}
    vp.set_trig_mode("precise")
    try:
        for v in (0, lists):
            _lib.LIB.vp_set_kernel_variant(0, v)
            y = torch.zeros(n, PX, H, device="cuda")
            vp._CU.forward_z0(xt, y, a)
            err[v] = float(np.sqrt(np.mean((y.cpu().numpy().astype(np.float64) - want) ** 2)))
    finally:
        _lib.LIB.vp_set_kernel_variant(0, 0)
        vp.set_trig_mode("reference")
    assert err[0] <= 1.1 * err[lists]
