"""The transposes of the z_order 2 path: tile edges and remainders on both axes,
rows in float4 or not on either side, pad heights, adding and storing, against
the z_order 0 call on transposed arrays, bit for bit."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests.common import lin, seeded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [32, 33, 63, 64, 65, 130])
@pytest.mark.parametrize("SY,SX,n,PX", [(8, 8, 16, 8), (9, 7, 13, 11), (33, 31, 7, 65),
                                        (16, 20, 21, 19)])
def test_z2_is_z0_transposed(SY, SX, n, PX, H):
    a = torch.tensor(lin(n, -0.2, 3.3), device="cuda")
    x2, y2 = (torch.tensor(seeded(s, 95 + i), device="cuda")
              for i, s in enumerate([(H, SY, SX), (H, n, PX)]))
    Hp = (H + 3) // 4 * 4
    x0, y0 = torch.zeros(SY, SX, Hp, device="cuda"), torch.zeros(n, PX, Hp, device="cuda")
    x0[..., :H] = x2.permute(1, 2, 0)
    y0[..., :H] = y2.permute(1, 2, 0)
    for forward, in2, in0, like2, like0 in ((True, x2, x0, y2, y0), (False, y2, y0, x2, x0)):
        ref = vp._CU.project_store(forward, 0, in0, torch.empty_like(like0), a)
        ref = ref[..., :H].permute(2, 0, 1)
        stored = vp._CU.project_store(forward, 2, in2, torch.empty_like(like2), a)
        assert torch.equal(stored, ref)
        added = like2.clone()
        (vp._CU.forward_z2 if forward else vp._CU.backward_z2)(in2, added, a)
        assert torch.equal(added, like2 + ref)
