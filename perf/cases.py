"""Performance cases: the calls a user of the framework makes, from the smallest to the largest.

``listed()`` are fixed cases, ``draw(rng)`` gives more of the same ranges.  ``prepare`` makes
seeded inputs and the plans or modules a program keeps, ``run`` is one pass through the public
entry points, ``work`` the bytes and operations such a pass cannot do without, and ``exact``
the same outputs in 64 bits by plain torch (None where that takes too long).
"""
import dataclasses
import math

import numpy as np
import torch

from fastcone_b200 import _lib, autograd, fastcone, nn, ops
from fastcone_b200.geometry import ConeGeometry
from fastcone_b200.phantom import random_ellipsoids
from fastcone_b200.sirt import SIRT

DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
WINDOWS = {"ramlak": _lib.FILTER_RAMLAK, "shepplogan": _lib.FILTER_SHEPPLOGAN,
           "cosramp": _lib.FILTER_COSRAMP, "gaussramp": _lib.FILTER_GAUSSRAMP}
EXACT_UPDATES = 6.0e10   # voxel-view updates, ray samples: beyond these exact() gives None
EXACT_SAMPLES = 3.0e10


def listed():
    return [
        # The small circular FDK problem (128^3, 180 views) with everything on the GPU and the
        # plan kept: a call of under a millisecond, a chip that the tiles hardly fill.
        dict(name="bp-small", op="bp", nx=128, ny=128, nz=128, W=192, H=128, views=180, D=500.0, pw=0.5,
             mode=2, dtype="f32"),
        # The large circular FDK problem (1024^3, 1440 views, 1536 x 1024 detector): the headline
        # workload, FP32 projections resident in device memory.
        dict(name="bp-large", op="bp", nx=1024, ny=1024, nz=1024, W=1536, H=1024, views=1440, D=2000.0, pw=0.8,
             mode=2, dtype="f32"),
        # A mid-size FDK problem with projections stored in BF16 (half the memory).
        dict(name="bp-mid-bf16", op="bp", nx=512, ny=512, nz=512, W=768, H=512, views=400, D=1000.0, pw=0.8,
             mode=2, dtype="bf16"),
        # An unweighted backprojection (the one for iterative methods) of a cropped scan: odd
        # volume and detector sizes, rows that no 16-byte boundary follows.
        dict(name="bp-odd", op="bp", nx=251, ny=237, nz=203, W=379, H=231, views=200, D=1000.0, pw=1.0,
             mode=0, dtype="f32"),
        # Helical Katsevich, 512 x 512 x 384, 4640 views on 736 x 64: the PI-window
        # backprojection with its plan, and the filtering of the same projections.
        dict(name="kats-bp", op="kats_bp", scale=1.0, vpt=1160),
        dict(name="kats-filter", op="kats_filter", scale=1.0, vpt=1160),
        # The cosine weight and Shepp-Logan filter of the large problem's projections.
        dict(name="filter-large", op="filter", views=1440, H=1024, W=1536, window="shepplogan", dtype="f32", cosw=True),
        # The drop-in fastcone.fbp on numpy arrays (the small problem), host to host.
        dict(name="fbp-host", op="fbp_host", n=128, W=192, H=128, views=180),
        # The smallest projection call: 64^3, 24 views, no plan kept (as autograd makes them).
        dict(name="project-small", op="project", nx=64, ny=64, nz=64, W=96, H=64, views=24, D=250.0, pw=1.0),
        # A data term ||A x - y||^2 and its gradient for a batch of 256^3 volumes.
        dict(name="loss-grad", op="loss_grad", batch=2, nx=256, ny=256, nz=256, W=384, H=256, views=180, D=1000.0, pw=1.0),
        # Training one 3x3x3 convolution layer of the learned reconstruction on a 256^3 volume:
        # output, input gradient, weight and bias gradients.
        dict(name="conv-train", op="conv", nx=256, ny=256, nz=256, relu=True),
        # SIRT iterations of the sparse-view problem (256^3, 90 views), from zero.
        dict(name="sirt", op="sirt", nx=256, ny=256, nz=256, W=384, H=256, views=90, D=1000.0, pw=1.0, iters=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["bp", "bp", "bp", "kats_bp", "kats_filter", "filter", "filter", "fbp_host", "project",
                     "loss_grad", "conv", "sirt"])
    if op == "bp":
        n = _log(rng, 48, 640)
        c = dict(op=op, nx=n, ny=max(16, int(n * rng.uniform(0.7, 1.1))), nz=max(8, int(n * rng.uniform(0.5, 1.1))),
                 pw=round(rng.uniform(0.5, 1.1), 2), D=float(int(n * rng.uniform(1.9, 4.0)) + 16),
                 mode=rng.choice([0, 1, 2, 2]), dtype=rng.choice(["f32", "f32", "bf16", "f16"]), views=_log(rng, 30, 720))
        c["W"] = int(1.45 * n / c["pw"] * rng.uniform(0.8, 1.1))
        c["H"] = int(1.2 * c["nz"] / c["pw"] * rng.uniform(0.8, 1.1))
        if rng.random() < 0.5:   # half the scanners have widths of whole 16-byte rows
            c["W"] = (c["W"] + 7) // 8 * 8
        return c
    if op in ("kats_bp", "kats_filter"):
        return dict(op=op, scale=round(math.exp(rng.uniform(math.log(0.12), math.log(0.8))), 3),
                    vpt=_log(rng, 150, 1000))
    if op == "filter":
        c = dict(op=op, views=_log(rng, 16, 400), H=_log(rng, 16, 1024), W=_log(rng, 48, 2048),
                 window=rng.choice(["ramlak", "shepplogan", "ramlak", "cosramp", "gaussramp"]),
                 dtype=rng.choice(["f32", "f32", "bf16", "f16"]))
        c["cosw"] = c["window"] in ("ramlak", "shepplogan") and rng.random() < 0.8
        return c
    if op == "fbp_host":
        n = 16 * _log(rng, 2, 16)
        return dict(op=op, n=n, W=n * 3 // 2, H=n, views=_log(rng, 24, 360))
    if op == "conv":
        return dict(op=op, nx=_log(rng, 24, 288), ny=_log(rng, 24, 288), nz=_log(rng, 16, 256), relu=rng.random() < 0.7)
    n = _log(rng, 32, 288 if op == "project" else 224)
    c = dict(op=op, nx=n, ny=n, nz=max(8, int(n * rng.uniform(0.5, 1.0))), W=int(1.5 * n), D=float(4 * n), pw=1.0,
             views=_log(rng, 16, 180))
    c["H"] = c["nz"]
    if rng.random() < 0.6:       # rows of whole 16-byte groups, as most volumes have
        c["nx"] = c["ny"] = (n + 3) // 4 * 4
    if op == "loss_grad":
        c["batch"] = rng.choice([1, 2, 3])
    if op == "sirt":
        c["iters"] = rng.choice([2, 3, 5])
    return c


# ------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _geom(c, norm=None):
    n = c["views"]
    ang = (np.arange(n, dtype=np.float64) * (2 * math.pi / n)).astype(np.float32)
    return ConeGeometry((c["nx"], c["ny"], c["nz"]), (c["W"], c["H"]), ang, c["D"], c["pw"],
                        norm=None if norm is None else np.full(n, norm, np.float32))


def _helix(c, pi_window):
    """The helical problem scaled by ``scale``: pitch 80, radius 1140, pw 1.096 voxels at 1."""
    s = c["scale"]
    n = max(32, int(512 * s)) // 2 * 2
    W = max(32, int(736 * s)) // 4 * 4
    H = max(8, int(64 * s))
    return ConeGeometry.helical((n, n, n * 3 // 4), 0.5 / s, (W, H), 1.0 / s, 570.0, 1040.0, 4, c["vpt"], 40.0,
                                pi_window=pi_window)


def _kats_norm(g):
    dlam = (float(g.angles[-1]) - float(g.angles[0])) / (g.nviews - 1)
    return abs(dlam) / (2 * math.pi * g.D)


def _line_integrals(shape, gen, seed, half=(0.5, 0.9)):
    """Projections as a scanner gives them, all >= 0: a smooth object shadow, whose half-width
    in each view is drawn from ``half`` (1: the whole detector), and noise that grows with it."""
    n, H, W = shape
    r = np.random.default_rng(seed)
    w = torch.linspace(-1, 1, W, device="cuda")
    h = torch.linspace(-1, 1, H, device="cuda")
    a = torch.tensor(r.uniform(*half, n), device="cuda", dtype=torch.float32)
    o = torch.tensor(r.uniform(-0.1, 0.1, n), device="cuda", dtype=torch.float32)
    p = torch.empty(shape, device="cuda")
    for t in range(n):
        q = (1 - ((w - o[t]) / a[t]) ** 2)[None, :] - 0.3 * (h ** 2)[:, None]
        torch.sqrt(q.clamp_(min=0), out=p[t])
    p.mul_(3.0)
    for t in range(0, n, 64):
        k = p[t:t + 64]
        k.mul_(torch.randn(k.shape, device="cuda", generator=gen).mul_(0.02).add_(1.0))
    return p


def _volume(c, gen, seed):
    vol = ops.phantom((c["nx"], c["ny"], c["nz"]), random_ellipsoids(10, (c["nx"], c["ny"], c["nz"]), seed))
    return vol.add_(torch.randn(vol.shape, device="cuda", generator=gen).mul_(0.01))


def prepare(case, seed):
    c, gen, op = case, _gen(seed), case["op"]
    s = {"case": c}
    if op == "bp":
        g = _geom(c, 1.0 / c["views"])
        s["proj"] = torch.empty(g.proj_shape, device="cuda", dtype=DT[c["dtype"]])
        for t in range(0, c["views"], 64):   # filtered projections: zero mean
            k = s["proj"][t:t + 64]
            k.copy_(torch.randn(k.shape, device="cuda", generator=gen))
        s["vol"] = torch.zeros(g.vol_shape, device="cuda")
        s["plan"] = ops.BackprojectPlan(g, mode=c["mode"], dtype=DT[c["dtype"]])
    elif op == "kats_bp":
        g = _helix(c, True)
        g = g.with_norm(np.full(g.nviews, _kats_norm(g), np.float32))
        s["proj"] = torch.randn(g.proj_shape, device="cuda", generator=gen)
        s["vol"] = torch.zeros(g.vol_shape, device="cuda")
        s["plan"] = ops.BackprojectPlan(g, mode=_lib.MODE_KATSEVICH)
    elif op == "kats_filter":
        g = _helix(c, False)
        s["proj"] = _line_integrals(g.proj_shape, gen, seed)
        s["out"] = torch.empty_like(s["proj"])
        s["plan"] = ops.KatsevichPlan(g)
    elif op == "filter":
        shape = (c["views"], c["H"], c["W"])
        s["proj"] = _line_integrals(shape, gen, seed)
        s["out"] = torch.empty(shape, device="cuda", dtype=DT[c["dtype"]])
        s["z"] = np.full(c["views"], c["H"] / 2.0, np.float32)
        s["D"] = 4.0 * c["W"] / 3.0
        s["plan"] = ops.FilterPlan(shape, out_dtype=DT[c["dtype"]], window=WINDOWS[c["window"]])
    elif op == "fbp_host":
        n, views = c["n"], c["views"]
        s["sino"] = _line_integrals((views, c["H"], c["W"]), gen, seed).cpu().numpy()
        s["proj"] = np.empty_like(s["sino"])
        s["vol"] = np.zeros((n, n, n), np.float32)
        s["angles"] = (np.arange(views) * (2 * math.pi / views)).astype(np.float32)
        s["z"] = np.full(views, n / 2.0, np.float32)
    elif op == "conv":
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        torch.manual_seed(seed)
        s["layer"] = nn.Conv3d(16, 16, relu=c["relu"]).cuda()
        with torch.no_grad():
            s["layer"].bias.uniform_(-0.1, 0.1)
        # activations after a ReLU; incoming gradients of both signs
        s["x"] = torch.randn((nz, ny, 2, nx, 8), device="cuda", generator=gen).relu_().to(torch.bfloat16).requires_grad_()
        s["gy"] = torch.randn((nz, ny, 2, nx, 8), device="cuda", generator=gen).to(torch.bfloat16)
    else:
        g = s["geom"] = _geom(c)
        if op == "project":
            s["vol"] = _volume(c, gen, seed)
        elif op == "loss_grad":
            s["x"] = torch.stack([_volume(c, gen, seed * 16 + b) for b in range(c["batch"])]).requires_grad_()
            s["y"] = torch.rand((c["batch"],) + g.proj_shape, device="cuda", generator=gen).mul_(0.5 * c["nx"])
        else:
            s["sirt"] = SIRT(g)
            # an object inside the volume: its shadow ends before the rays that graze the volume
            s["y"] = _line_integrals(g.proj_shape, gen, seed, half=(0.3, 0.5))
    return s


def run(s):
    op = s["case"]["op"]
    if op in ("bp", "kats_bp"):
        return s["plan"](s["proj"], s["vol"].zero_())
    if op == "kats_filter":
        return s["plan"](s["proj"], out=s["out"])
    if op == "filter":
        c = s["case"]
        if c["cosw"]:
            return s["plan"](s["proj"], zorigin=s["z"], D=s["D"], out=s["out"])
        return s["plan"](s["proj"], cosine_weight=False, out=s["out"])
    if op == "fbp_host":
        n = s["case"]["n"]
        np.copyto(s["proj"], s["sino"])   # the next scan arrives in the program's array
        s["vol"].fill(0.0)
        fastcone.fbp(s["vol"], s["proj"], s["angles"], 500.0 * n / 128, s["z"], pixelWidth=0.5)
        return s["vol"], s["proj"]
    if op == "conv":
        layer = s["layer"]
        y = layer(s["x"])
        gx, dw, db = torch.autograd.grad(y, [s["x"], layer.weight, layer.bias], s["gy"])
        return {"y": y.detach(), "gx": gx, "dw": dw, "db": db}
    if op == "project":
        return ops.project(s["vol"], s["geom"], method=_lib.PROJ_EXPLICIT)
    if op == "loss_grad":
        p = autograd.project(s["x"], s["geom"])
        loss = ((p - s["y"]) ** 2).sum()
        grad, = torch.autograd.grad(loss, s["x"])
        return {"proj": p.detach(), "grad": grad}
    return s["sirt"].run(s["y"], iters=s["case"]["iters"])


# --------------------------------------------------------------------------- work
def _samples(c):
    """Ray samples inside the volume, about: the mean chord over the detector's rays."""
    return 0.6 * c["views"] * c["W"] * c["H"] * c["nx"]


def work(case):
    c, op = case, case["op"]
    if op == "bp":
        v, p = c["nx"] * c["ny"] * c["nz"], c["views"] * c["H"] * c["W"]
        return {"bytes": 4 * v + p * (4 if c["dtype"] == "f32" else 2), "flops": 8.0 * v * c["views"]}
    if op in ("kats_bp", "kats_filter"):
        g = _helix(c, False)
        p = g.nviews * g.det_wh[0] * g.det_wh[1]
        if op == "kats_filter":   # two transforms of each row's 2 W points, and the other passes
            return {"bytes": 8 * p, "flops": p * (2 * 2 * 2.5 * 2 * math.log2(2 * g.det_wh[0]) + 30)}
        v = int(np.prod(g.vol_shape))
        # a voxel sees about half a turn of the views
        return {"bytes": 4 * p + 4 * v, "flops": 8.0 * v * 0.5 * c["vpt"]}
    if op == "filter":
        p = c["views"] * c["H"] * c["W"]
        return {"bytes": p * (4 + (4 if c["dtype"] == "f32" else 2)), "flops": p * (2 * 2.5 * 2 * math.log2(2 * c["W"]) + 6)}
    if op == "fbp_host":
        v, p = c["n"] ** 3, c["views"] * c["H"] * c["W"]
        return {"bytes": 4 * v + 8 * p, "flops": 8.0 * v * c["views"] + p * (10 * math.log2(2 * c["W"]) + 6)}
    v = c["nx"] * c["ny"] * c["nz"]
    if op == "conv":   # x, y, gy read and written, gx; three products of 27 taps x 16 x 16
        return {"bytes": v * 16 * 2 * 4, "flops": 3.0 * 2 * 27 * 16 * 16 * v}
    p = c["views"] * c["H"] * c["W"]
    if op == "project":
        return {"bytes": 4 * v + 4 * p, "flops": 15.0 * _samples(c)}
    if op == "loss_grad":
        return {"bytes": c["batch"] * (8 * v + 8 * p), "flops": c["batch"] * 38.0 * _samples(c)}
    return {"bytes": 4 * v + 4 * p, "flops": c["iters"] * (15.0 * _samples(c) + 8.0 * v * c["views"])}


# ------------------------------------------------------------------ 64-bit values
F64 = torch.float64


def _bp64(proj, vol_xyz, det_wh, angles, D, pw, hmid, norm, mode, pitch=0.0):
    """Voxel-driven backprojection in 64 bits; pitch != 0: over each voxel's PI interval."""
    nx, ny, nz = vol_xyz
    W, H = det_wh
    x = (torch.arange(nx, device="cuda", dtype=F64) - nx // 2)[None, :]
    y = (torch.arange(ny, device="cuda", dtype=F64) - ny // 2)[:, None]
    z = torch.arange(nz, device="cuda", dtype=F64) - nz // 2
    out = torch.zeros((nz, ny, nx), device="cuda", dtype=F64)
    turn = float(angles[-1]) - float(angles[0])
    sgn = -1.0 if (turn >= 0) == (pitch >= 0) else 1.0
    nzb = max(1, min(nz, int(2.0e7 / (nx * ny))))
    for t in range(len(angles)):
        ca, sa = math.cos(float(angles[t])), math.sin(float(angles[t]))
        hmp = float(hmid[t]) - nz // 2
        U = D / (D + x * ca + y * sa)
        wm = (y * ca - x * sa) * U
        w = wm / pw + W // 2
        wi = torch.floor(w)
        fw = w - wi
        wi = wi.long().clamp(-2, W) + 2
        pad = torch.zeros((H + 4, W + 4), device="cuda", dtype=F64)
        pad[2:-2, 2:-2] = proj[t].to(F64)
        flat = pad.reshape(-1)
        wt = float(norm[t]) * U ** mode
        for z0 in range(0, nz, nzb):
            zz = (z[z0:z0 + nzb] - hmp)[:, None, None]
            hm = zz * U
            h = hm / pw + H // 2
            hi = torch.floor(h)
            fh = h - hi
            i = (hi.long().clamp(-2, H) + 2) * (W + 4) + wi
            a = torch.lerp(flat[i], flat[(i + 1).clamp_(max=flat.numel() - 1)], fw.expand_as(fh))
            i += W + 4
            b = torch.lerp(flat[i.clamp(max=flat.numel() - 1)], flat[(i + 1).clamp_(max=flat.numel() - 1)], fw.expand_as(fh))
            val = torch.lerp(a, b, fh) * wt
            if pitch != 0.0:
                u = sgn * wm / D
                q = pitch / (2 * math.pi) * (1 + u * u)
                at = torch.atan(u)
                val = val * ((hm <= q * (0.5 * math.pi - at)) & (hm >= -q * (0.5 * math.pi + at)))
            out[z0:z0 + nzb] += val
    return out


def _rays64(c, t):
    """Source and unit directions of view t's pixels, in voxel-index coordinates."""
    a = float(np.float32(t * (2 * math.pi / c["views"])))
    ca, sa = math.cos(a), math.sin(a)
    o = torch.tensor([c["nx"] // 2, c["ny"] // 2, c["nz"] // 2], device="cuda", dtype=F64)
    hmp = c["nz"] / 2.0 - c["nz"] // 2
    w = (torch.arange(c["W"], device="cuda", dtype=F64) - c["W"] // 2) * c["pw"]
    h = (torch.arange(c["H"], device="cuda", dtype=F64) - c["H"] // 2) * c["pw"] + hmp
    src = torch.tensor([-c["D"] * ca, -c["D"] * sa, hmp], device="cuda", dtype=F64)
    p = torch.stack(torch.broadcast_tensors(-sa * w[None, :], ca * w[None, :], h[:, None]), -1)
    d = p - src
    return src + o, (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)


def _project64(c, vol=None, proj=None):
    """A vol (vol given) or A^T proj: every integer distance from the source, trilinear."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    sx, sy, sz = 1, nx + 4, (nx + 4) * (ny + 4)
    pad = torch.zeros((nz + 4, ny + 4, nx + 4), device="cuda", dtype=F64)
    if vol is not None:
        pad[2:-2, 2:-2, 2:-2] = vol.to(F64)
    flat = pad.reshape(-1)
    r = 0.5 * math.sqrt(nx * nx + ny * ny + nz * nz) + 4
    out = torch.zeros((c["views"], c["H"] * c["W"]), device="cuda", dtype=F64)
    for t in range(c["views"]):
        src, d = _rays64(c, t)
        reach = 0.5 * math.hypot(c["W"], c["H"]) * c["pw"]
        # the volume's bounding sphere along any ray of the detector
        m0, m1 = int(c["D"] - r) - 2, int(math.hypot(c["D"], reach) + r) + 2
        step = max(1, int(4.0e7 / d.shape[0]))
        for a in range(max(0, m0), m1 + 1, step):
            m = torch.arange(a, min(a + step, m1 + 1), device="cuda", dtype=F64)[:, None]
            idx = torch.zeros((m.shape[0], d.shape[0]), device="cuda", dtype=torch.int64)
            f = []
            ok = torch.ones_like(idx, dtype=torch.bool)
            for k, (n, st) in enumerate(((nx, sx), (ny, sy), (nz, sz))):
                q = src[k] + m * d[:, k]
                i = torch.floor(q)
                f.append(q - i)
                ok &= (i >= -1) & (i <= n - 1)
                idx += (i.clamp_(-1, n - 1).long() + 2) * st
            if vol is not None:
                e = [torch.lerp(torch.lerp(flat[idx + dz], flat[idx + dz + 1], f[0]),
                                torch.lerp(flat[idx + dz + sy], flat[idx + dz + sy + 1], f[0]), f[1]) for dz in (0, sz)]
                out[t] += (torch.lerp(e[0], e[1], f[2]) * ok).sum(0)
            else:
                v = proj[t].reshape(-1).to(F64)[None, :] * ok
                for b in range(8):
                    wgt = v
                    for k in range(3):
                        wgt = wgt * (f[k] if (b >> k) & 1 else 1 - f[k])
                    flat.index_add_(0, (idx + (b & 1) * sx + (b >> 1 & 1) * sy + (b >> 2) * sz).reshape(-1), wgt.reshape(-1))
    if vol is not None:
        return out.reshape(c["views"], c["H"], c["W"])
    return pad[2:-2, 2:-2, 2:-2].clone()


def _ramp64(proj, window, cosw, z, D):
    n, H, W = proj.shape
    L = 2 * W if window in ("ramlak", "shepplogan") else W
    k = torch.arange(L // 2 + 1, device="cuda", dtype=F64)
    if L == 2 * W:
        f = k / L
        f[0] = 0.125 / L
        if window == "shepplogan":
            x = math.pi * k[1:] / L
            f[1:] = f[1:] * torch.sin(x) / x
        f = f * math.pi
    else:
        f = k / W
        if window == "cosramp":
            f = f * torch.cos(0.5 * f * math.pi / W)
        else:
            f = torch.where(k + 0.5 * W <= W - 1, f * torch.exp(-0.5 * ((k + 0.5) / (0.125 * W)) ** 2), torch.zeros_like(f))
    out = torch.empty(proj.shape, device="cuda", dtype=F64)
    ww = torch.arange(W, device="cuda", dtype=F64) - W / 2.0
    for t in range(n):
        p = proj[t].to(F64)
        if cosw:
            hh = torch.arange(H, device="cuda", dtype=F64)[:, None] - float(z[t])
            p = p * (D / torch.sqrt(D * D + hh * hh + ww * ww))
        out[t] = torch.fft.irfft(torch.fft.rfft(p, n=L, dim=-1) * f, n=L, dim=-1)[:, :W]
    return out


def _kats64(proj, g):
    """Katsevich filtering on the flat detector through the axis (Noo, Pack & Heuscher 2003)."""
    n, H, W = proj.shape
    D, pw, P = float(np.float32(g.D)), float(np.float32(g.pw)), float(np.float32(g.helical_pitch))
    su = -1.0
    dl = (float(g.angles[-1]) - float(g.angles[0])) / (n - 1)
    u = su * (torch.arange(W, device="cuda", dtype=F64) - W // 2) * pw
    v = (torch.arange(H, device="cuda", dtype=F64) - H // 2) * pw
    K = 2 * H
    am = math.atan(float(u.abs().max()) / D)
    psi = -math.pi / 2 - am + (math.pi + 2 * am) * torch.arange(K, device="cuda", dtype=F64) / (K - 1)
    cot = torch.where(psi.abs() < 1e-12, torch.ones_like(psi), psi / torch.tan(psi))
    vk = (P / (2 * math.pi)) * (psi[:, None] + cot[:, None] * u[None, :] / D)       # [K, W], rising in k
    x = (vk - v[0]) / pw
    j0 = x.floor().long().clamp(0, H - 2)
    fa = (x - j0) * ((vk >= v[0]) & (vk <= v[-1]))
    keep = ((vk >= v[0]) & (vk <= v[-1])).to(F64)
    b = torch.searchsorted(vk.t().contiguous(), v[None, :].expand(W, H).contiguous(), right=True).t() - 1   # [H, W]
    k0 = b.clamp(0, K - 2)
    lo, hi = torch.gather(vk, 0, k0), torch.gather(vk, 0, k0 + 1)
    fb = ((v[:, None] - lo) / (hi - lo)).clamp(0, 1)
    m = torch.arange(-(W - 1), W, device="cuda")
    ker = torch.where(m % 2 != 0, 2.0 / (math.pi * m.to(F64)), torch.zeros(1, device="cuda", dtype=F64))
    L = 4 * W
    kern = torch.zeros(L, device="cuda", dtype=F64)
    kern[m % L] = ker
    ks = torch.fft.rfft(kern)
    q2 = u * u + D * D
    out = torch.empty(proj.shape, device="cuda", dtype=F64)
    for t in range(n):
        a, e = max(0, t - 1), min(n - 1, t + 1)
        c = proj[t].to(F64)
        g1 = (proj[e].to(F64) - proj[a].to(F64)) / ((e - a) * dl)
        g1 = g1 + q2 / D * (torch.gradient(c, dim=1)[0] / (su * pw)) + u * v[:, None] / D * (torch.gradient(c, dim=0)[0] / pw)
        g2 = g1 * D / torch.sqrt(q2 + v[:, None] ** 2)
        r0, r1 = torch.gather(g2, 0, j0), torch.gather(g2, 0, j0 + 1)
        g3 = torch.lerp(r0, r1, fa) * keep
        g4 = su * torch.fft.irfft(torch.fft.rfft(g3, n=L, dim=-1) * ks, n=L, dim=-1)[:, :W]
        out[t] = torch.lerp(torch.gather(g4, 0, k0), torch.gather(g4, 0, k0 + 1), fb)
    return out


def _conv64(x, wk):
    """sum over taps of the shifted x [nz, ny, nx, cin] times wk[tap] [cin, cout]."""
    nz, ny, nx, _ = x.shape
    y = torch.zeros((nz, ny, nx, wk.shape[2]), device="cuda", dtype=F64)
    for t, (src, dst) in enumerate(_shifts(nz, ny, nx)):
        y[dst] += x[src] @ wk[t]
    return y


def _shifts(nz, ny, nx):
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                s = tuple(slice(max(0, d), n + min(0, d)) for d, n in ((dz, nz), (dy, ny), (dx, nx)))
                t = tuple(slice(max(0, -d), n + min(0, -d)) for d, n in ((dz, nz), (dy, ny), (dx, nx)))
                yield s, t


def exact(case, seed):
    c, op = case, case["op"]
    if op in ("bp", "kats_bp"):
        g = _geom(c) if op == "bp" else _helix(c, True)
        if float(np.prod(g.vol_shape)) * g.nviews > EXACT_UPDATES:
            return None
        s = prepare(c, seed)
        p = s["plan"].geom
        return _bp64(s["proj"], p.vol_xyz, p.det_wh, p.angles, float(np.float32(p.D)), float(np.float32(p.pw)), p.hmid,
                     p.norm, c["mode"] if op == "bp" else 1, float(np.float32(p.helical_pitch)) if op == "kats_bp" else 0.0)
    if op == "kats_filter":
        return _kats64(prepare(c, seed)["proj"], _helix(c, False))
    if op == "filter":
        s = prepare(c, seed)
        return _ramp64(s["proj"], c["window"], c["cosw"], s["z"], float(np.float32(s["D"])))
    if op == "fbp_host":
        # only where the reference's sub-problem windows, which this entry point follows, hold
        # the whole footprint
        if (c["n"], c["W"], c["H"]) != (128, 192, 128):
            return None
        s = prepare(c, seed)
        f = _ramp64(torch.from_numpy(s["sino"]).cuda(), "ramlak", True, s["z"], 500.0)
        n = c["n"]
        vol = _bp64(f, (n, n, n), (c["W"], c["H"]), s["angles"], 500.0, 0.5, s["z"],
                    np.full(c["views"], 1.0 / c["views"]), 2)
        return vol, f
    if op == "conv":
        s = prepare(c, seed)
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        to = lambda t: t.detach().to(F64).permute(0, 1, 3, 2, 4).reshape(nz, ny, nx, 16)  # noqa: E731
        back = lambda t: t.reshape(nz, ny, nx, 2, 8).permute(0, 1, 3, 2, 4).contiguous()  # noqa: E731
        w = s["layer"].weight.detach().to(torch.bfloat16).to(F64)
        wk = w.permute(2, 3, 4, 1, 0).reshape(27, 16, 16)      # [tap][in][out]
        x = to(s["x"])
        y = _conv64(x, wk) + s["layer"].bias.detach().to(F64)
        gy = to(s["gy"])
        if c["relu"]:
            gy *= y > 0
            y.clamp_(min=0)
        y = back(y)
        gx = back(_conv64(gy, wk.flip(0).transpose(1, 2)))
        dw = torch.stack([x[a].reshape(-1, 16).t() @ gy[b].reshape(-1, 16) for a, b in _shifts(nz, ny, nx)])
        return {"y": y, "gx": gx, "dw": dw.reshape(3, 3, 3, 16, 16).permute(4, 3, 0, 1, 2).contiguous(),
                "db": gy.sum(dim=(0, 1, 2))}
    passes = {"project": 1, "loss_grad": 3 * c.get("batch", 0), "sirt": c.get("iters", 0) + 1}[op]
    if passes * _samples(c) / 0.6 > EXACT_SAMPLES:
        return None
    s = prepare(c, seed)
    if op == "project":
        return _project64(c, vol=s["vol"])
    if op == "loss_grad":
        x = s["x"].detach()
        p = torch.stack([_project64(c, vol=v) for v in x])
        g = torch.stack([_project64(c, proj=2 * (p[b] - s["y"][b].to(F64))) for b in range(c["batch"])])
        return {"proj": p, "grad": g}
    g = dataclasses.replace(s["geom"])
    B = lambda p: _bp64(p, g.vol_xyz, g.det_wh, g.angles, c["D"], c["pw"], g.hmid, np.ones(g.nviews), 0)  # noqa: E731
    inv = lambda t: torch.where(t > 1e-6, 1.0 / t.clamp_min(1e-6), torch.zeros_like(t))  # noqa: E731
    ones = torch.ones(g.vol_shape, device="cuda", dtype=F64)
    R, C = inv(_project64(c, vol=ones)), inv(B(torch.ones(g.proj_shape, device="cuda", dtype=F64)))
    x, y = torch.zeros_like(ones), s["y"].to(F64)
    for _ in range(c["iters"]):
        x = (x + C * B((y - _project64(c, vol=x)) * R)).clamp_(min=0)
    return x
