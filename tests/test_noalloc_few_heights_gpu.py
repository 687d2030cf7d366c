"""vp_forward_z2_noalloc below 32 heights: one kernel, no scratch.  Such calls share
nothing, may be a process's first under stream capture, and have no size limit."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest
import torch

from oracle import oracle
from tests import tolerances as tol
from tests.common import lin, rel_err, seeded
from voxelproj_gb300 import _lib

pytestmark = pytest.mark.gpu


def _call(fn, x, y, a):
    before = _lib.LIB.vp_launch_count()
    stream = torch.cuda.current_stream().cuda_stream
    assert fn(x.data_ptr(), *x.shape, y.data_ptr(), *y.shape, a.data_ptr(), a.numel(), 0,
              stream) == _lib.VP_OK
    return _lib.LIB.vp_launch_count() - before


@pytest.mark.parametrize("H", [1, 4, 5, 8, 13, 31])
def test_one_kernel(H):
    SY, SX, n, PX = 45, 38, 33, 52
    ang = lin(n, -0.3, 3.3)
    x, y0 = seeded((H, SY, SX), 61), seeded((H, n, PX), 62)
    y = torch.tensor(y0, device="cuda")
    assert _call(_lib.LIB.vp_forward_z2_noalloc, torch.tensor(x, device="cuda"), y,
                 torch.tensor(ang, device="cuda")) == 1
    assert rel_err(y.cpu().numpy() - y0, oracle.forward(x, ang, PX, 2)) <= tol.ref_vs_fp64(PX)


def test_beyond_the_array():
    H, S, n = 29, 720, 40
    assert _lib.LIB.vp_z2_workspace_bytes(H, S, S, H, n, S) > _lib.VP_NOALLOC_SCRATCH_BYTES
    x = torch.randn(H, S, S, device="cuda")
    a = torch.tensor(lin(n), device="cuda")
    y, want = (torch.zeros(H, n, S, device="cuda") for _ in range(2))
    assert _call(_lib.LIB.vp_forward_z2_noalloc, x, y, a) == 1
    _call(_lib.LIB.vp_forward_z2, x, want, a)
    # two float32 evaluations of one bin coordinate
    assert float((y - want).abs().max() / want.abs().max()) <= 2 * tol.ref_vs_fp64(S)


_FIRST_UNDER_CAPTURE = r"""
import os, sys
import torch
sys.path.insert(0, sys.argv[1])
from voxelproj_gb300 import _lib
x, y = torch.randn(13, 20, 20, device="cuda"), torch.zeros(13, 12, 20, device="cuda")
a = torch.linspace(0, 3, 12).cuda()
torch.cuda.synchronize()
s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
    st = _lib.LIB.vp_forward_z2_noalloc(x.data_ptr(), *x.shape, y.data_ptr(), *y.shape,
                                        a.data_ptr(), 12, 0, s.cuda_stream)
assert st == 0, (st, _lib.LIB.vp_last_cuda_error())
assert _lib.LIB.vp_launch_count() == 1
g.replay()
torch.cuda.synchronize()
assert float(y.abs().sum()) > 0
print("ok", flush=True)
os._exit(0)
"""


def test_first_call_under_capture():
    root = Path(__file__).resolve().parent.parent
    res = subprocess.run([sys.executable, "-c", _FIRST_UNDER_CAPTURE, str(root)], cwd=root,
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "ok" in res.stdout, res.stdout + res.stderr
