"""The banded 4-height forward (vp_fp_band.cuh): runs per warp 8, 4, 3, 2, 1, lines
split over four warps or not, partial height chunks and remainders, outputs
written by float4 and by single heights, narrow and wide angles of both signs,
windows over every edge of the volume."""

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

# around the angles where the bands change from 4 to 5 voxels per bin
EDGES = np.float32([0, 0.6, 0.61, 0.62, 0.64, 0.785398, 0.93, 0.96, 1.5707964, 2.2, 2.3561945,
                    2.5, 3.1415927, 4.0, 5.4, -0.7])


@pytest.mark.parametrize("H", [5, 8, 16, 17, 32, 33, 40, 41, 64, 65, 100, 128, 130, 161, 192, 257, 420])
@pytest.mark.parametrize("geom", [(9, 6, 11), (40, 33, 50), (70, 130, 64)],
                         ids=lambda g: "x".join(map(str, g)))
@pytest.mark.parametrize("many", [False, True])
def test_band_matches_oracle(geom, H, many):
    """many: enough angles that the blocks fill a wave and no lines are split."""
    SY, SX, PX = geom
    if many and (H > 41 or geom != (40, 33, 50)):
        pytest.skip("one geometry is enough")
    ang = np.concatenate([EDGES, lin(2500 if many else 21, -0.3, 6.4)])
    x, y0 = seeded((SY, SX, H), 81), seeded((len(ang), PX, H), 82)
    y = torch.tensor(y0, device="cuda")
    vp._CU.forward_z0(torch.tensor(x, device="cuda"), y, torch.tensor(ang, device="cuda"))
    err = rel_err(y.cpu().numpy() - y0, oracle.forward(x, ang, PX, 0))
    assert err <= tol.ref_vs_fp64(max(SY, SX, PX))


@pytest.mark.parametrize("H", [12, 32, 40, 64, 128])
def test_band_equals_candidate_lists(H):
    """Unsplit and in one slab the sums are those of the candidate lists, bit for
    bit (variant 10: the same bins per warp and lines)."""
    SY, SX, PX = 60, 50, 70
    n = 1400 if H == 12 else 800
    a = torch.tensor(lin(n, -0.3, 6.4), device="cuda")
    x = torch.tensor(seeded((SY, SX, H), 83), device="cuda")
    outs = []
    for v in (0, 10):
        _lib.LIB.vp_set_kernel_variant(0, v)
        try:
            y = torch.zeros(n, PX, H, device="cuda")
            vp._CU.forward_z0(x, y, a)
            outs.append(y)
        finally:
            _lib.LIB.vp_set_kernel_variant(0, 0)
    assert torch.equal(*outs)


@pytest.mark.parametrize("H,n", [(8, 9), (64, 9), (128, 2000)])
def test_non_finite_voxels_reach_their_bins_only(H, n):
    """An infinite voxel reaches the bins that its three weights go to and no
    others: as with the candidate lists."""
    SY, SX, PX = 30, 30, 30
    a = torch.tensor(lin(n), device="cuda")
    x = torch.randn(SY, SX, H, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    x[11, 17, 3] = float("inf")
    x[20, 5, 6] = float("nan")
    outs = []
    for v in (0, 10):
        _lib.LIB.vp_set_kernel_variant(0, v)
        try:
            y = torch.zeros(n, PX, H, device="cuda")
            vp._CU.forward_z0(x, y, a)
            outs.append(y)
        finally:
            _lib.LIB.vp_set_kernel_variant(0, 0)
    f = [torch.isfinite(o) for o in outs]
    assert torch.equal(*f)
    assert not f[0].all() and f[0][..., :3].all() and f[0][..., 7:].all()
    assert torch.allclose(outs[0][f[0]], outs[1][f[1]], rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("H", [5, 13, 31])
def test_z2_few_heights_with_and_without_workspace(H):
    """vp_forward_z2_ws from 5 to 31 heights: transposed with a workspace, without
    it (too small) on its own kernel; both are the operator."""
    SY, SX, n, PX = 33, 29, 40, 45
    ang = lin(n, -0.3, 3.3)
    x = seeded((H, SY, SX), 84)
    xt, a = torch.tensor(x, device="cuda"), torch.tensor(ang, device="cuda")
    need = _lib.LIB.vp_z2_workspace_bytes(H, SY, SX, H, n, PX)
    assert need > 0
    ws = torch.full(((need + 3) // 4,), float("nan"), device="cuda")
    ref = oracle.forward(x, ang, PX, 2)
    for nbytes in (need, 0):
        y = torch.zeros(H, n, PX, device="cuda")
        st = _lib.LIB.vp_forward_z2_ws(xt.data_ptr(), *xt.shape, y.data_ptr(), *y.shape,
                                       a.data_ptr(), n, 0, ws.data_ptr(), nbytes,
                                       torch.cuda.current_stream().cuda_stream)
        assert st == _lib.VP_OK
        assert rel_err(y.cpu().numpy(), ref) <= tol.ref_vs_fp64(PX)
