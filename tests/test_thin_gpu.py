"""Projections of few heights (vp_thin.cu) against the oracle: heights per lane
1, 2, 4 and 8 with partial last chunks, both layouts, bins and voxels that are
not multiples of a warp, one to several chunks of lines, one and four voxels
per lane, angle sets with both minor axes and both signs of each step."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import voxelproj_gb300 as vp
from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded, x_shape, y_shape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trig", ["reference", "precise"])
@pytest.mark.parametrize("z", [0, 2])
@pytest.mark.parametrize("H", [1, 2, 3, 5, 8, 31])
@pytest.mark.parametrize("geom", [(1, 1, 5, 3), (33, 17, 40, 31), (70, 65, 37, 97),
                                  (19, 130, 60, 64)], ids=lambda g: "x".join(map(str, g)))
def test_thin_matches_oracle(geom, H, z, trig):
    SY, SX, n, PX = geom
    ang = lin(n, -0.3, 6.4)
    ang[:2] = [0.0, np.float32(np.pi / 2)]
    x, y = seeded(x_shape(z, SY, SX, H), 61), seeded(y_shape(z, n, PX, H), 62)
    vp.set_trig_mode(trig)
    try:
        yo, xo = torch.tensor(y, device="cuda"), torch.tensor(x, device="cuda")
        a = torch.tensor(ang, device="cuda")
        (vp._CU.forward_z0 if z == 0 else vp._CU.forward_z2)(torch.tensor(x, device="cuda"), yo, a)
        (vp._CU.backward_z0 if z == 0 else vp._CU.backward_z2)(torch.tensor(y, device="cuda"), xo, a)
    finally:
        vp.set_trig_mode("reference")
    N = max(SY, SX, PX)
    bound = tol.precise_vs_fp64(N) if trig == "precise" else tol.ref_vs_fp64(N)
    assert rel_err(yo.cpu().numpy() - y, oracle.forward(x, ang, PX, z)) <= bound
    assert rel_err(xo.cpu().numpy() - x, oracle.backward(y, ang, SY, SX, z)) <= bound


def test_large_slice_each_way():
    """Enough voxels for four per lane, and rows beyond the last group of four."""
    SY, SX, n, PX = 515, 260, 24, 300
    ang = lin(n, 0.1, 3.2)
    x, y = seeded((1, SY, SX), 63), seeded((1, n, PX), 64)
    ax = vp.forward(torch.tensor(x, device="cuda"), ang, (1, n, PX), z_order=2).cpu().numpy()
    aty = vp.backward(torch.tensor(y, device="cuda"), ang, (1, SY, SX), z_order=2).cpu().numpy()
    bound = tol.ref_vs_fp64(SY)
    assert rel_err(ax, oracle.forward(x, ang, PX, 2)) <= bound
    assert rel_err(aty, oracle.backward(y, ang, SY, SX, 2)) <= bound


def test_voxels_outside_a_bin_do_not_reach_it():
    """An infinite voxel makes infinite only the bins whose rays meet it."""
    x = torch.zeros(1, 40, 40, device="cuda")
    x[0, 20, 11] = float("inf")
    y = vp.forward(x, lin(30), (1, 30, 40), z_order=2)
    assert not torch.isnan(y).any()
    hit = torch.isinf(y).sum(dim=2)
    assert int(hit.max()) <= 3 and int(hit.min()) >= 1


@pytest.mark.parametrize("n", [360, 251])
@pytest.mark.parametrize("H", [1, 2, 4])
def test_large_slices_match_many_heights(H, n):
    """512 x 512 slices at many angles (every rounding of an edge against a tile's border):
    the thin forward against the transposed path of 8 heights."""
    g = torch.Generator(device="cuda").manual_seed(9)
    a = torch.tensor(lin(n, 0.0, 3.1415927), device="cuda")
    x = torch.randn(8, 512, 500, device="cuda", generator=g)
    want = torch.zeros(8, n, 520, device="cuda")
    vp._CU.forward_z2(x, want, a)
    y = torch.zeros(H, n, 520, device="cuda")
    vp._CU.forward_z2(x[:H].contiguous(), y, a)
    # two float32 evaluations of one bin coordinate: the bound of either against 64 bits
    err = (y - want[:H]).abs().max() / want.abs().max()
    assert err <= 2 * tol.ref_vs_fp64(520)
