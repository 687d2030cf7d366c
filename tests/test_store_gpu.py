"""vp_project_store: out = A in or A^T in whatever out held, equal to the adding
calls on zeros bit for bit; heights of out past the input's, and outputs that
the operator does not reach, are zero."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests.common import lin, seeded, x_shape, y_shape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [0, 2])
@pytest.mark.parametrize("Hx,Hy", [(1, 1), (7, 7), (20, 20), (64, 64), (45, 45), (260, 260),
                                   (8, 12), (40, 33), (3, 5)])
def test_store_equals_adding_to_zeros(Hx, Hy, z):
    SY, SX, n, PX = 30, 26, 35, 41
    a = torch.tensor(lin(n, -0.2, 3.3), device="cuda")
    x = torch.tensor(seeded(x_shape(z, SY, SX, Hx), 91), device="cuda")
    y = torch.tensor(seeded(y_shape(z, n, PX, Hy), 92), device="cuda")
    calls = vp._CU
    for forward, inp, like, add in (
            (True, x, y, calls.forward_z0 if z == 0 else calls.forward_z2),
            (False, y, x, calls.backward_z0 if z == 0 else calls.backward_z2)):
        ref = torch.zeros_like(like)
        add(inp, ref, a)
        out = torch.full_like(like, float("nan"))
        assert calls.project_store(forward, z, inp, out, a) is out
        assert torch.equal(out, ref)


@pytest.mark.parametrize("shape", [(0, 26, 8), (30, 26, 0)])
def test_empty_problems_store_zeros(shape):
    a = torch.tensor(lin(5), device="cuda")
    x = torch.zeros(shape, device="cuda")
    out = torch.full((5, 12, 8), float("nan"), device="cuda")
    vp._CU.project_store(True, 0, x, out, a)
    assert not out.any()
