"""Calls on pageable host arrays touch nothing past them: arrays whose last byte lies
before an inaccessible page, in a process of their own."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

_SCRIPT = r"""
import ctypes, mmap, os, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
import voxelproj_gb300 as vp

libc = ctypes.CDLL(None)
libc.mmap.restype = ctypes.c_void_p
libc.mmap.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                      ctypes.c_long]
libc.mprotect.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
PAGE = mmap.PAGESIZE

def guarded(values):
    size = -(-values.nbytes // PAGE) * PAGE
    p = libc.mmap(None, size + 256 * PAGE, mmap.PROT_READ | mmap.PROT_WRITE,
                  mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS, -1, 0)
    assert p not in (None, ctypes.c_void_p(-1).value)
    assert libc.mprotect(p + size, 256 * PAGE, 0) == 0
    a = np.ctypeslib.as_array((ctypes.c_float * values.size).from_address(p + size - values.nbytes))
    a = a.reshape(values.shape)
    a[...] = values
    return a

z, H, SY, SX, n = (int(v) for v in sys.argv[2:7])
ang = np.linspace(-0.2, 3.2, n).astype(np.float32)
rng = np.random.default_rng(1)
x = rng.standard_normal((SY, SX, H) if z == 0 else (H, SY, SX)).astype(np.float32)
y = rng.standard_normal((n, SX, H) if z == 0 else (H, n, SX)).astype(np.float32)
out = guarded(y)
vp.forward(guarded(x), guarded(ang), out, z_order=z)
want = y.copy()
vp.forward(torch.from_numpy(x).pin_memory(), ang, torch.from_numpy(want), z_order=z)
assert np.abs(out - want).max() <= 1e-5 * np.abs(want).max()
out = guarded(x)
vp.backward(guarded(y), guarded(ang), out, z_order=z)
want = x.copy()
vp.backward(torch.from_numpy(y).pin_memory(), ang, torch.from_numpy(want), z_order=z)
assert np.abs(out - want).max() <= 1e-5 * np.abs(want).max()
print("ok", flush=True)
os._exit(0)
"""


@pytest.mark.parametrize("z,H,SY,SX,n", [
    (2, 257, 199, 199, 20),  # the adjoint's last chunk is one height, in row slabs
    (2, 513, 160, 150, 12), (2, 300, 150, 160, 30), (2, 66, 320, 300, 20), (2, 33, 90, 80, 40),
    (2, 13, 60, 70, 21), (2, 1, 50, 60, 20), (0, 203, 90, 100, 70), (0, 3, 60, 70, 30),
    (0, 128, 140, 150, 40),
])
def test_nothing_past_the_arrays(z, H, SY, SX, n):
    root = Path(__file__).resolve().parent.parent
    res = subprocess.run([sys.executable, "-c", _SCRIPT, str(root), *map(str, (z, H, SY, SX, n))],
                         cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "ok" in res.stdout, (res.returncode, res.stdout + res.stderr)
