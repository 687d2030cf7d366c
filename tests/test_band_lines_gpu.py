"""The banded forward leaves out the lines that its runs of bins do not see: the sums
of the candidate lists bit for bit on volumes and detectors of very different
extents, and no time for bins that see nothing."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests.common import lin, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


def _forward(x, y, a, variant=0):
    _lib.LIB.vp_set_kernel_variant(0, variant)
    try:
        vp._CU.forward_z0(x, y, a)
    finally:
        _lib.LIB.vp_set_kernel_variant(0, 0)
    return y


@pytest.mark.parametrize("H", [8, 32, 40, 64, 100])
@pytest.mark.parametrize("SY,SX,PX", [(5, 61, 400), (61, 5, 90), (1, 30, 300), (30, 30, 500),
                                      (2, 2, 350), (64, 20, 13)])
def test_equals_candidate_lists(SY, SX, PX, H):
    """Enough angles that no lines are split; one slab (variant 10: the same bins per warp)."""
    n = 7600 // max(1, PX // 16)
    a = torch.cat([torch.tensor(lin(n, -0.4, 6.6)), torch.tensor([0.0, 1.5707964, 0.785398, 1e-6])])
    a = a.cuda()
    x = torch.tensor(seeded((SY, SX, H), 41), device="cuda")
    y = [_forward(x, torch.zeros(len(a), PX, H, device="cuda"), a, v) for v in (0, 10)]
    assert torch.equal(*y)


def test_bins_off_the_volume_take_no_time():
    """Four times the bins, none of the new ones on the volume: with every line taken
    the time was about that of their number."""

    def time(PX):
        a = torch.tensor(lin(400, 1.3, 1.8), device="cuda")
        x, y = torch.randn(40, 300, 48, device="cuda"), torch.zeros(400, PX, 48, device="cuda")
        best = float("inf")
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(5):
                vp._CU.forward_z0(x, y, a)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert time(1200) <= 2.0 * time(300)
