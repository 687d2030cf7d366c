"""Timed cases of the projector pair, through the package's public entry points.

A case is a dict of plain values:

  op     "forward"   y += A x        (voxelproj_gb300.forward)
         "backward"  x += A^T y      (voxelproj_gb300.backward)
         "gradient"  r = A x - b and A^T r of 0.5 |A x - b|^2, through autograd
         "batch"     A and A^T of `count` uneven cubes in one batch plan
  z      memory order: 0 (heights fastest) or 2 (heights slowest)
  SY, SX volume rows and columns; H heights; n angles over [0, pi); PX bins
  out    "add": into a container that the caller keeps; "new": allocated by the call
  trig   "reference" or "precise" per-angle constants
  data   "device": CUDA tensors; "host": page-locked host tensors in and out

Volumes are phantoms of ellipsoids with noise, sinograms are noise residuals:
what a reconstruction passes to A and A^T.
"""

import math

import numpy as np
import torch

import voxelproj_gb300 as vp
from voxelproj_gb300.autograd import project
from voxelproj_gb300.batch import Batch

# A drawn case's voxel x angle updates.  Odd heights and few heights cost more
# per update than whole float4 heights; with this bound they stay below the
# largest listed case all the same.
MOST_UPDATES = 1.0e10


def _case(name, op, z, SY, SX, H, n, PX, out="add", trig="reference", data="device"):
    return {"name": name, "op": op, "z": z, "SY": SY, "SX": SX, "H": H, "n": n, "PX": PX,
            "out": out, "trig": trig, "data": data}


def listed():
    return [
        # a small served request (sides from 32): one iteration's A and A^T
        _case("small_gradient", "gradient", 0, 32, 32, 32, 128, 32, out="new"),
        # a single slice, as in 2-D reconstruction, each direction
        _case("slice_forward_z2", "forward", 2, 512, 512, 1, 360, 512, out="new"),
        _case("slice_backward_z2", "backward", 2, 512, 512, 1, 360, 512, out="new"),
        # a thin stack of slices (a fan of detector rows) in the slices-first order
        _case("stack_gradient_z2", "gradient", 2, 384, 384, 16, 180, 384, out="new"),
        # the small cube of the benchmark tables
        _case("cube128_gradient", "gradient", 0, 128, 128, 128, 192, 128, out="new"),
        # a cropped scan: odd sizes, a detector wider than the volume, heights
        # that are not whole float4, each direction
        _case("ragged_forward", "forward", 0, 301, 257, 203, 181, 397),
        _case("ragged_backward", "backward", 0, 301, 257, 203, 181, 397, trig="precise"),
        # one step of the differentiable reconstruction, slices first
        _case("cube256_gradient_z2", "gradient", 2, 256, 256, 256, 360, 256, out="new"),
        # arrays that live in host memory, copies included
        _case("cube256_host_forward", "forward", 0, 256, 256, 256, 360, 256, data="host"),
        # the headline size, each direction; more angles than the usual 192 on
        # the way back
        _case("cube512_forward", "forward", 0, 512, 512, 512, 192, 512),
        _case("cube512_backward", "backward", 0, 512, 512, 512, 1024, 512),
        # uneven requests in one submission
        {"name": "batch_uneven", "op": "batch", "count": 8, "low": 32, "high": 160,
         "n_low": 90, "n_high": 360, "sizes": 2026},
    ]


def _spread(rng, low, high):
    """A whole number of [low, high], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.random()
    if kind < 0.08:
        return {"op": "batch", "count": rng.randint(3, 10), "low": 4 * rng.randint(6, 12),
                "high": 4 * rng.randint(16, 40), "n_low": rng.randint(45, 90),
                "n_high": rng.randint(91, 400), "sizes": rng.randint(0, 1 << 20)}
    op = rng.choice(["forward", "backward", "gradient"])
    z = rng.choice([0, 2])
    SX = _spread(rng, 24, 512)
    SY = SX if rng.random() < 0.5 else _spread(rng, max(24, SX // 2), min(512, 2 * SX))
    thick = rng.random()
    if thick < 0.15:
        H = 1  # one slice
    elif thick < 0.35:
        H = _spread(rng, 2, 31)  # a thin stack
    else:
        H = _spread(rng, 32, 512)
        if rng.random() < 0.6:
            H = (H + 3) // 4 * 4
    n = _spread(rng, 30, 1024)
    side = max(SY, SX)
    width = rng.random()
    if width < 0.5:
        PX = side  # the default
    elif width < 0.8:
        PX = int(math.ceil(math.hypot(SY, SX))) + rng.randint(0, 8)  # the whole footprint
    else:
        PX = rng.randint(max(16, side // 2), side)  # a cut detector
    while float(SY) * SX * H * n > MOST_UPDATES:
        n = max(30, n // 2)
        if n == 30:
            H = max(1, H // 2)
    return {"op": op, "z": z, "SY": SY, "SX": SX, "H": H, "n": n, "PX": PX,
            "out": "new" if op == "gradient" else rng.choice(["add", "new"]),
            "trig": "precise" if rng.random() < 0.2 else "reference",
            "data": "host" if op != "gradient" and rng.random() < 0.15 else "device"}


# --------------------------------------------------------------------------
# inputs


def _angles(n):
    return np.linspace(0.0, np.pi, n, endpoint=False).astype(np.float32)


def _shapes(c):
    vol = (c["SY"], c["SX"], c["H"]) if c["z"] == 0 else (c["H"], c["SY"], c["SX"])
    sino = (c["n"], c["PX"], c["H"]) if c["z"] == 0 else (c["H"], c["n"], c["PX"])
    return vol, sino


def _cubes(c):
    """(side, angles) of each cube of a batch; sides in whole float4."""
    rng = np.random.default_rng(c["sizes"])
    return [(int(4 * rng.integers(c["low"] // 4, c["high"] // 4 + 1)),
             int(rng.integers(c["n_low"], c["n_high"] + 1))) for _ in range(c["count"])]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _phantom(shape, seed):
    """A few ellipsoids of densities around one, with noise."""
    dev = _device()
    rng = np.random.default_rng(int(seed))
    axes = [torch.linspace(-1.0, 1.0, s, device=dev) if s > 1 else torch.zeros(1, device=dev)
            for s in shape]
    x = 0.05 * torch.randn(shape, device=dev, generator=_generator(seed))
    for _ in range(6):
        centre, half = rng.uniform(-0.6, 0.6, 3), rng.uniform(0.15, 0.6, 3)
        density = float(rng.uniform(0.3, 1.0))
        q = [((t - float(m)) / float(a)) ** 2 for t, m, a in zip(axes, centre, half)]
        inside = (q[0][:, None, None] + q[1][None, :, None]) + q[2][None, None, :] <= 1.0
        x += density * inside
    return x


def _residual(shape, seed):
    return torch.randn(shape, device=_device(), generator=_generator(int(seed) + 7919))


def _container(shape, seed):
    return 0.1 * torch.randn(shape, device=_device(), generator=_generator(int(seed) + 104729))


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _inputs(c, seed):
    """(x or None, y or None, container or None) of a projection case, on the device."""
    vol, sino = _shapes(c)
    x = _phantom(vol, seed) if c["op"] != "backward" else None
    y = _residual(sino, seed) if c["op"] != "forward" else None
    out = None
    if c["out"] == "add":
        out = _container(sino if c["op"] == "forward" else vol, seed)
    return x, y, out


def _cube_inputs(c, seed):
    return [(n, _phantom((s, s, s), seed + 31 * k), _residual((n, s, s), seed + 31 * k))
            for k, (s, n) in enumerate(_cubes(c))]


def prepare(case, seed):
    c = case
    if c["op"] == "batch":
        problems, outs = [], []
        for n, x, y in _cube_inputs(c, seed):
            a = torch.from_numpy(_angles(n)).cuda()
            ax, aty = torch.zeros_like(y), torch.zeros_like(x)
            problems += [("forward", x, ax, a), ("backward", y, aty, a)]
            outs += [ax, aty]
        return {"case": c, "batch": Batch(problems), "outs": outs}
    x, y, out = _inputs(c, seed)
    if c["data"] == "host":
        x, y, out = (None if t is None else _pinned(t) for t in (x, y, out))
        angles = _angles(c["n"])
    else:
        angles = torch.from_numpy(_angles(c["n"])).cuda()
    return {"case": c, "x": x, "y": y, "out": out, "angles": angles}


def run(state):
    c = state["case"]
    if c["op"] == "batch":
        state["batch"].run()
        return state["outs"]
    precise = c["trig"] == "precise"
    if precise:
        vp.set_trig_mode("precise")
    try:
        vol, sino = _shapes(c)
        if c["op"] == "forward":
            out = state["out"] if state["out"] is not None else sino
            return vp.forward(state["x"], state["angles"], out, z_order=c["z"])
        if c["op"] == "backward":
            out = state["out"] if state["out"] is not None else vol
            return vp.backward(state["y"], state["angles"], out, z_order=c["z"])
        x = state["x"].detach().requires_grad_(True)
        r = project(x, state["angles"], c["PX"], c["z"]) - state["y"]
        # the gradient of 0.5 r.r is A^T r
        grad, = torch.autograd.grad(r, x, grad_outputs=r.detach())
        return {"residual": r.detach(), "gradient": grad}
    finally:
        if precise:
            vp.set_trig_mode("reference")


# --------------------------------------------------------------------------
# what a pass cannot do without


def _nonzeros(SY, SX, n, PX):
    """Nonzero weights of A per height, from a sample of the grid: a voxel
    covers 1 + |cos| + |sin| bins on average, where they are on the detector."""
    a = _angles(n).astype(np.float64)
    a = a[:: max(1, n // 64)]
    yy = np.linspace(-(SY - 1) / 2, (SY - 1) / 2, min(SY, 64))
    xx = np.linspace(-(SX - 1) / 2, (SX - 1) / 2, min(SX, 64))
    xp = np.cos(a)[:, None, None] * xx[None, None, :] + np.sin(a)[:, None, None] * yy[None, :, None]
    on = (np.abs(xp) <= PX / 2).mean(axis=(1, 2))
    return float(SY) * SX * n * float(np.mean(on * (1 + np.abs(np.cos(a)) + np.abs(np.sin(a)))))


def _work_of(op, SY, SX, H, n, PX, out):
    vol, sino = 4.0 * SY * SX * H, 4.0 * n * PX * H
    flops = 2.0 * _nonzeros(SY, SX, n, PX) * H
    if op == "gradient":  # x and b in, r and the gradient out
        return 2 * vol + 2 * sino, 2 * flops
    src, dst = (vol, sino) if op == "forward" else (sino, vol)
    return src + (2 if out == "add" else 1) * dst, flops


def work(case):
    c = case
    if c["op"] == "batch":
        parts = [_work_of(op, s, s, s, n, s, "add") for s, n in _cubes(c)
                 for op in ("forward", "backward")]
    else:
        parts = [_work_of(c["op"], c["SY"], c["SX"], c["H"], c["n"], c["PX"], c["out"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# --------------------------------------------------------------------------
# the operator in 64 bits


def _cdf(t, a, b, coeff, cd):
    """Area of the unit voxel's trapezoidal footprint left of t."""
    left = cd * (t + b) ** 2
    mid = coeff * (a + b) + 2 * coeff * t
    right = 1 - cd * (b - t) ** 2
    v = torch.where(t < a, torch.where(t < -a, left, mid), right)
    return torch.where(t <= -b, torch.zeros_like(v), torch.where(t >= b, torch.ones_like(v), v))


def _footprints(angles, SY, SX, PX):
    """Bins and weights, each (angles, SY * SX, 3), and whether each bin is on
    the detector."""
    a64 = torch.from_numpy(angles.astype(np.float64)).to(_device())[:, None, None]
    c, s = torch.cos(a64), torch.sin(a64)
    p, m = (0.5 * (c + s)).abs(), (0.5 * (c - s)).abs()
    a, b = torch.minimum(p, m), torch.maximum(p, m)
    coeff = 0.5 / (a + b)
    cd = torch.where(b > a, coeff / torch.where(b > a, b - a, torch.ones_like(a)),
                     torch.zeros_like(a))
    yy = torch.arange(SY, device=_device(), dtype=torch.float64) - (SY - 1) / 2
    xx = torch.arange(SX, device=_device(), dtype=torch.float64) - (SX - 1) / 2
    xp = c * xx[None, None, :] + s * yy[None, :, None] + (PX - 1) / 2
    r = torch.round(xp)
    f0, f1 = _cdf(r - xp - 0.5, a, b, coeff, cd), _cdf(r - xp + 0.5, a, b, coeff, cd)
    n = len(angles)
    w = torch.stack([f0, f1 - f0, 1 - f1], dim=-1).reshape(n, SY * SX, 3)
    bins = (r.to(torch.int64)[..., None]
            + torch.arange(-1, 2, device=_device())).reshape(n, SY * SX, 3)
    return bins, w, (bins >= 0) & (bins < PX)


def _matrices(angles, SY, SX, PX):
    """(first angle, count, A of these angles as a sparse (count * PX, SY * SX) matrix)."""
    step = max(1, (6 << 20) // (3 * SY * SX))
    for k in range(0, len(angles), step):
        part = angles[k:k + step]
        bins, w, on = _footprints(part, SY, SX, PX)
        row = bins + PX * torch.arange(len(part), device=_device())[:, None, None]
        col = torch.arange(SY * SX, device=_device())[None, :, None].expand_as(bins)
        yield k, len(part), row[on], col[on], w[on]


def _exact_forward(x, angles, PX):
    """A x in 64 bits; x (SY, SX, H)."""
    SY, SX, H = x.shape
    flat = x.double().reshape(SY * SX, H)
    y = torch.empty(len(angles), PX, H, dtype=torch.float64, device=x.device)
    for k, m, row, col, w in _matrices(angles, SY, SX, PX):
        A = torch.sparse_coo_tensor(torch.stack([row, col]), w, (m * PX, SY * SX))
        y[k:k + m] = torch.sparse.mm(A, flat).reshape(m, PX, H)
    return y


def _exact_backward(y, angles, SY, SX):
    """A^T y in 64 bits; y (n, PX, H)."""
    n, PX, H = y.shape
    x = torch.zeros(SY * SX, H, dtype=torch.float64, device=y.device)
    for k, m, row, col, w in _matrices(angles, SY, SX, PX):
        AT = torch.sparse_coo_tensor(torch.stack([col, row]), w, (SY * SX, m * PX))
        x += torch.sparse.mm(AT, y[k:k + m].double().reshape(m * PX, H))
    return x.reshape(SY, SX, H)


def _to_z0(t, z):
    return t if z == 0 else t.permute(1, 2, 0).contiguous()


def _from_z0(t, z):
    return t if z == 0 else t.permute(2, 0, 1).contiguous()


def exact(case, seed):
    c = case
    if c["op"] == "batch":
        outs = []
        for n, x, y in _cube_inputs(c, seed):
            outs += [_exact_forward(x, _angles(n), y.shape[1]),
                     _exact_backward(y, _angles(n), x.shape[0], x.shape[1])]
        return outs
    x, y, out = _inputs(c, seed)
    z, angles = c["z"], _angles(c["n"])
    if c["op"] == "forward":
        v = _from_z0(_exact_forward(_to_z0(x, z), angles, c["PX"]), z)
        return v if out is None else v + out.double()
    if c["op"] == "backward":
        v = _from_z0(_exact_backward(_to_z0(y, z), angles, c["SY"], c["SX"]), z)
        return v if out is None else v + out.double()
    r = _exact_forward(_to_z0(x, z), angles, c["PX"]) - _to_z0(y, z).double()
    g = _exact_backward(r, angles, c["SY"], c["SX"])
    return {"residual": _from_z0(r, z), "gradient": _from_z0(g, z)}
