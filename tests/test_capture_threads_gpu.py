"""Calls that take memory of their own (padded rows in z_order 0, transposes in z_order 2)
leave a stream capture of another thread alone: the first call of a process, which
makes the pool, and the next ones."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

_SCRIPT = r"""
import os, sys, threading
import torch
sys.path.insert(0, sys.argv[1])
import voxelproj_gb300 as vp
from voxelproj_gb300 import _lib

z = int(sys.argv[2])
n, S = 20, 40
a = torch.linspace(0, 3, n).cuda()
x0 = torch.randn(S, S, 64, device="cuda")
y0 = torch.zeros(n, S, 64, device="cuda")
vp._CU.forward_z0(x0, y0, a)  # no scratch
want0 = y0.clone()
y0.zero_()
calls = []
for s, H in ((S, 45 if z == 0 else 13), (400, 47 if z == 0 else 15)):
    x = torch.randn(*((s, s, H) if z == 0 else (H, s, s)), device="cuda")
    y = torch.zeros(*((n, s, H) if z == 0 else (H, n, s)), device="cuda")
    calls.append((x, y))
torch.cuda.synchronize()
other = torch.cuda.Stream()
status = []

def work():
    fn = _lib.LIB.vp_forward_z0 if z == 0 else _lib.LIB.vp_forward_z2
    for x, y in calls:
        status.append(fn(x.data_ptr(), *x.shape, y.data_ptr(), *y.shape, a.data_ptr(), n, 0,
                         other.cuda_stream))

capture, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.stream(capture), torch.cuda.graph(graph, stream=capture):
    vp._CU.forward_z0(x0, y0, a)
    t = threading.Thread(target=work)
    t.start()
    t.join()
assert status == [0, 0], (status, _lib.LIB.vp_last_cuda_error())
graph.replay()
torch.cuda.synchronize()
assert torch.equal(y0, want0)
for x, y in calls:
    ref = torch.zeros_like(y)
    (vp._CU.forward_z0 if z == 0 else vp._CU.forward_z2)(x, ref, a)
    assert float((y - ref).abs().max()) <= 1e-4 * float(ref.abs().max())
print("ok", flush=True)
os._exit(0)
"""


@pytest.mark.parametrize("z", [0, 2])
def test_capture_of_another_thread_survives(z):
    root = Path(__file__).resolve().parent.parent
    res = subprocess.run([sys.executable, "-c", _SCRIPT, str(root), str(z)], cwd=root,
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "ok" in res.stdout, res.stdout + res.stderr
