"""The run adjoint's block orders (tile_order in vp_bp_runs.cuh): a sinogram large
enough for bands of tiles equals the same heights in pieces small enough for row
order, bit for bit (every voxel sums its angles in the same order), single, in
row slabs from host arrays and batched."""

from __future__ import annotations

import pytest
import torch

import voxelproj_gb300 as vp
from tests.common import lin
from voxelproj_gb300.batch import Batch

pytestmark = pytest.mark.gpu

PX = 150


# 69 and 20 tile rows (bands of 20 + 20 + 20 + 9 and 64 + 5, and one whole band); columns in
# whole tiles or not; 4 and 8 heights per lane, a rest of 4 each
@pytest.mark.parametrize("SY,SX", [(275, 36), (274, 37), (80, 8), (9, 300)])
@pytest.mark.parametrize("H,n", [(128, 2100), (256, 1100), (320, 2100)])
def test_bands_equal_rows(SY, SX, H, n):
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.tensor(lin(n, -0.3, 6.4), device="cuda")
    y = torch.randn(n, PX, H, device="cuda", generator=g)
    x0 = torch.randn(SY, SX, H, device="cuda", generator=g)
    assert n * PX * min(H, 256) * 4 > 144 << 20  # the large order
    want = torch.empty_like(x0)
    for h in range(0, H, 32):
        part = x0[..., h:h + 32].contiguous()
        vp._CU.backward_z0(y[..., h:h + 32].contiguous(), part, a)
        want[..., h:h + 32] = part
    x = x0.clone()
    vp._CU.backward_z0(y, x, a)
    assert torch.equal(x, want)
    x = x0.clone()
    b = Batch([("backward", y, x, a)])
    b.run()
    torch.cuda.synchronize()
    assert not b.error()
    b.close()
    assert torch.equal(x, want)


def test_host_row_slabs():
    SY, SX, H, n = 275, 36, 128, 2100
    g = torch.Generator().manual_seed(6)
    a = torch.tensor(lin(n, -0.3, 6.4))
    y = torch.randn(n, PX, H, generator=g)
    x0 = torch.randn(SY, SX, H, generator=g)
    want = x0.cuda()
    vp._CU.backward_z0(y.cuda(), want, a.cuda())
    x = x0.numpy().copy()
    vp.backward(y.numpy(), a.numpy(), x)
    # the host call sums a first share of the angles apart and adds its container
    # last: two orders of one float32 sum over n angles differ by about
    # 2 sqrt(n) 2^-24 = 6e-6 of the largest partial sum
    assert (torch.from_numpy(x) - want.cpu()).abs().max() <= 1e-5 * want.abs().max()
