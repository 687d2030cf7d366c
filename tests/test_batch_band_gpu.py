"""Batched forwards of the default variant: banded 4-height parts (all run counts
per warp, warps on neighbouring run sets or angles, 129 to 192 heights as two
parts on the slab plan of the 8-height form) equal the single-problem kernel
of VP_BATCH_FORWARD_DEFAULT bit for bit."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests.common import lin, seeded
from voxelproj_gb300 import _lib
from voxelproj_gb300.batch import FORWARD_DEFAULT, Batch

pytestmark = pytest.mark.gpu

GEOMS = [(20, 26, 31, 29), (50, 40, 13, 150)]  # SY, SX, angles, bins


@pytest.mark.parametrize("geoms,heights", [
    (GEOMS, (8, 16, 20, 32, 36, 40, 64, 100, 128)),
    (GEOMS, (132, 140, 192, 196, 400, 448)),
    ([(330, 320, 10, 300)], (160, 416)),  # several slabs
])
def test_default_equals_single_variant(geoms, heights):
    problems, outs = [], []
    for SY, SX, n, PX in geoms:
        a = torch.tensor(lin(n, -0.3, 3.4), device="cuda")
        for H in heights:
            x = torch.tensor(seeded((SY, SX, H), 97 + H), device="cuda")
            y = torch.tensor(seeded((n, PX, H), 98 + H), device="cuda")
            outs.append((x, y, y.clone(), a))
            problems.append(("forward", x, y, a))
    b = Batch(problems)
    b.run()
    torch.cuda.synchronize()
    assert not b.error()
    _lib.LIB.vp_set_kernel_variant(0, FORWARD_DEFAULT)
    try:
        for x, y, y0, a in outs:
            vp._CU.forward_z0(x, y0, a)
            assert torch.equal(y, y0)
    finally:
        _lib.LIB.vp_set_kernel_variant(0, 0)
    b.close()
