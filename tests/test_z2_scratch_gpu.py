"""z_order 2 scratch below 32 heights through Python: none for the adjoint, and a
forward that runs without it where there is no memory for it."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests import tolerances as tol
from tests.common import lin

pytestmark = pytest.mark.gpu


def _peak(fn):
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    fn()
    torch.cuda.synchronize()
    return torch.cuda.max_memory_allocated() - before


@pytest.mark.parametrize("H", [4, 5, 17, 31])
def test_adjoint_takes_no_scratch(H):
    a = torch.tensor(lin(20), device="cuda")
    y, x = torch.randn(H, 20, 150, device="cuda"), torch.zeros(H, 150, 150, device="cuda")
    assert _peak(lambda: vp._CU.backward_z2(y, x, a)) == 0
    assert _peak(lambda: vp._CU.project_store(False, 2, y, x, a)) == 0


@pytest.mark.parametrize("store", [False, True])
def test_forward_without_memory_for_its_scratch(store):
    H, S, n = 31, 512, 24
    a = torch.tensor(lin(n), device="cuda")
    x, y = torch.randn(H, S, S, device="cuda"), torch.zeros(H, n, S, device="cuda")
    want = torch.zeros_like(y)
    vp._CU.forward_z2(x, want, a)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    # room for a few MB more than torch holds now; the scratch is 34 MB
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / total)
    try:
        if store:
            vp._CU.project_store(True, 2, x, y, a)
        else:
            vp._CU.forward_z2(x, y, a)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    # (either kernel may have run: two float32 evaluations of one bin coordinate)
    assert float((y - want).abs().max() / want.abs().max()) <= 2 * tol.ref_vs_fp64(S)
