"""Timed cases of the reconstruction path, each one pass through the package's public entry points.

``listed()`` are the standing cases, ``draw()`` more of the same ranges; ``prepare()`` makes what a program holds
before the call (images, angles, contexts, plans), ``run()`` is the pass and returns every output, ``work()`` the
bytes and operations a pass cannot do without, ``exact()`` the same outputs in 64 bits from plain torch and numpy.

In ``exact()`` the gridding follows the definition of the operations: rotation matrices, slice coordinates, the
interpolation table and its index are REAL (they choose discrete table entries), every sum and transform is 64-bit.
The trilinear, FBS and bilinear operators are continuous in the sample position, so theirs are 64-bit too.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spider_b200 import autograd as ag
from spider_b200 import ops

DEV = "cuda:0"


def listed():
    return [
        # one small BP 3F from start to end, grids and plans included: a quick look at a class average's few views
        {"name": "bp3f_call_64", "kind": "bp_call", "nx": 64, "images": 200},
        # RB 32F of one chunk at 128^3, the usual half-set refinement round: alignment by RTSQ, +-3 px shifts
        {"name": "rb32f_128", "kind": "bp", "nx": 128, "images": 4096, "grids": 2, "inplane": True, "bf16": False,
         "host": False, "sym": 1},
        # BP 32F at 256^3, images resident in HBM: the large box, two half-set grids
        {"name": "bp32f_256", "kind": "bp", "nx": 256, "images": 2048, "grids": 2, "inplane": False, "bf16": False,
         "host": False, "sym": 1},
        # the same box with BF16 spectra, images streamed from pinned host memory
        {"name": "bp32f_256_bf16_host", "kind": "bp", "nx": 256, "images": 1024, "grids": 2, "inplane": False,
         "bf16": True, "host": True, "sym": 1},
        # a box of odd size with D3 symmetry: six slices per image and SYMVOL
        {"name": "bp3f_147_d3", "kind": "bp", "nx": 147, "images": 300, "grids": 1, "inplane": False, "bf16": False,
         "host": False, "sym": 6},
        # several classes of different box sizes through one insertion launch per round
        {"name": "multiclass_4", "kind": "multi", "boxes": "96,128,160,224", "images": 4000},
        # reprojection of a small volume at a few angles: latency and host work
        {"name": "pj3q_call_64", "kind": "pj3q", "nx": 64, "images": 50},
        # differentiable projection, forward and backward, at a box whose packed volume exceeds the L2 limits
        {"name": "pj3q_grad_192", "kind": "pj3q_grad", "nx": 192, "images": 400},
        # PJ 3F (FBS interpolation)
        {"name": "pj3f_96", "kind": "pj3f", "nx": 96, "images": 500},
        # differentiable central-slice extraction, forward and backward, FP32, at a box that is no power of two
        {"name": "fslice_grad_150", "kind": "fs_grad", "nx": 150, "images": 800},
        # a whole regularised reconstruction on the central-slice pair: staging, FP64 CG, volume
        {"name": "fslice_cg_128", "kind": "fs_cg", "nx": 128, "images": 2000, "iters": 4},
        # BP CG from host arrays in the default precision: setup and three iterations
        {"name": "bpcg_128", "kind": "bpcg", "nx": 128, "images": 1000, "iters": 3},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fill(nx, grids=1, sym=1):
    """Images enough that nearly every Fourier voxel is covered, as a reconstruction's are: with fewer, voxels whose
    weight comes near NRMW2's threshold of 0.1 are kept or dropped by the last bit of a REAL sum."""
    return max(20, 3 * nx * grids // sym)


def draw(rng):
    kind = rng.choice(["bp_call", "bp", "bp", "bp", "multi", "pj3q", "pj3q_grad", "pj3f", "fs_grad", "fs_cg", "bpcg"])
    if kind == "bp_call":
        nx = _logint(rng, 24, 96)
        return {"kind": kind, "nx": nx, "images": _logint(rng, _fill(nx), 600)}
    if kind == "bp":
        nx = _logint(rng, 32, 256)
        sym = rng.choice([1, 1, 1, 2, 4, 6])
        inplane = rng.random() < 0.25
        grids = rng.choice([1, 2])
        least, most = _fill(nx, grids, sym), min(4096, int(2000 * (256 / nx) ** 2 / sym))
        return {"kind": kind, "nx": nx, "images": _logint(rng, least, max(least, most)), "grids": grids,
                "inplane": inplane, "bf16": rng.random() < 0.3, "host": rng.random() < 0.3, "sym": sym}
    if kind == "multi":
        boxes = [_logint(rng, 32, 224) for _ in range(rng.randint(2, 5))]
        least = len(boxes) * _fill(max(boxes), 2)
        return {"kind": kind, "boxes": ",".join(map(str, boxes)), "images": _logint(rng, least, max(least, 4000))}
    if kind == "pj3q":
        return {"kind": kind, "nx": _logint(rng, 32, 160), "images": _logint(rng, 1, 400)}
    if kind == "pj3q_grad":
        nx = _logint(rng, 48, 256)
        return {"kind": kind, "nx": nx, "images": _logint(rng, 16, min(1500, int(350 * (192 / nx) ** 3)))}
    if kind == "pj3f":
        nx = _logint(rng, 32, 128)
        return {"kind": kind, "nx": nx, "images": _logint(rng, 10, min(1000, int(480 * (96 / nx) ** 3)))}
    if kind == "fs_grad":
        nx = _logint(rng, 48, 256)
        return {"kind": kind, "nx": nx, "images": _logint(rng, 16, min(3000, int(800 * (150 / nx) ** 2)))}
    if kind == "fs_cg":
        nx = _logint(rng, 32, 160)
        return {"kind": kind, "nx": nx, "images": _logint(rng, 50, min(3000, int(2000 * (128 / nx) ** 2))),
                "iters": rng.randint(2, 4)}
    nx = _logint(rng, 32, 144)
    return {"kind": "bpcg", "nx": nx, "images": _logint(rng, 30, min(1500, int(950 * (128 / nx) ** 3))),
            "iters": rng.randint(1, 3)}


# ---------------------------------------------------------------------------- inputs
def _cang(psi_theta_phi):
    """Rotation matrices [n, 9] float32 (DM(1..9)); pi is a REAL constant there."""
    a = np.asarray(psi_theta_phi, np.float32).astype(np.float64) * (float(np.float32(math.pi)) / 180.0)
    cp, sp, ct, st, cf, sf = (f(a[:, k]) for k in range(3) for f in (np.cos, np.sin))
    dm = np.stack([cf * ct * cp - sf * sp, sf * ct * cp + cf * sp, -st * cp, -cf * ct * sp - sf * cp,
                   -sf * ct * sp + cf * cp, st * sp, st * cf, st * sf, ct], 1)
    return dm.astype(np.float32)


def _angles(n, rng):
    psi, phi = rng.uniform(0.0, 360.0, n), rng.uniform(0.0, 360.0, n)
    theta = np.degrees(np.arccos(rng.uniform(-1.0, 1.0, n)))
    return np.stack([psi, theta, phi], 1).astype(np.float32)


def _blobs(nx, rng, nblobs=40):
    """Centres (x, y, z), sigmas and amplitudes of a phantom of Gaussian blobs."""
    c = rng.normal(size=(nblobs, 3))
    c *= (0.375 * nx * rng.uniform(0, 1, (nblobs, 1)) ** (1 / 3)) / np.linalg.norm(c, axis=1, keepdims=True)
    return c, rng.uniform(max(1.5, nx / 85), max(2.0, nx / 25), nblobs), rng.uniform(0.5, 1.0, nblobs)


def _gauss(pos, sigma, nx):
    g = torch.arange(nx, device=DEV, dtype=torch.float32) - nx // 2
    return torch.exp(-((g - pos[..., None]) ** 2) / (2 * sigma[:, None] ** 2))


def _images(nx, ang, blobs, seed, snr=0.1):
    """Projections of the blobs along the rotations (analytic) with white noise at the given SNR."""
    c, s, amp = (torch.as_tensor(v, device=DEV, dtype=torch.float32) for v in blobs)
    dm = torch.as_tensor(_cang(ang), device=DEV)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    out = torch.empty((len(ang), nx, nx), device=DEV)
    for a in range(0, len(ang), 512):
        d = dm[a:a + 512]
        ex = _gauss(d[:, 0:3] @ c.T, s, nx) * (amp * s * math.sqrt(2 * math.pi))[:, None]
        im = torch.bmm(_gauss(d[:, 3:6] @ c.T, s, nx).transpose(1, 2), ex)
        sd = (im.var(dim=(1, 2), keepdim=True) / snr).sqrt()
        out[a:a + 512] = im + sd * torch.randn(im.shape, device=DEV, generator=gen)
    return out


def _volume(nx, blobs, seed):
    c, s, amp = (torch.as_tensor(v, device=DEV, dtype=torch.float32) for v in blobs)
    ex, ey, ez = (_gauss(c[:, k], s, nx) for k in range(3))
    v = torch.einsum("b,bz,by,bx->zyx", amp, ez, ey, ex)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return v + 0.05 * torch.randn(v.shape, device=DEV, generator=gen)


# D2, D3 and C2 as SPIDER writes them in a symmetry document: (psi, theta, phi)
_SYM = {1: None, 2: [(0, 0, 0), (0, 0, 180)], 4: [(0, 0, 0), (0, 0, 180), (0, 180, 0), (0, 180, 180)],
        6: [(0, 0, 0), (0, 0, 120), (0, 0, 240), (0, 180, 0), (0, 180, 120), (0, 180, 240)]}


def _sym(n):
    return None if n == 1 else np.array(_SYM[n], np.float32)


def _bp_inputs(nx, n, rng, seed):
    ang = _angles(n, rng)
    return _images(nx, ang, _blobs(nx, rng), seed), ang, (rng.random(n) < 0.5).astype(np.uint8)


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    k = case["kind"]
    if k == "multi":
        boxes = [int(b) for b in case["boxes"].split(",")]
        which = rng.integers(0, len(boxes), case["images"])
        return {"classes": [_bp_inputs(b, max(1, int((which == i).sum())), rng, seed + i)
                            for i, b in enumerate(boxes)]}
    nx, n = case["nx"], case["images"]
    if k in ("bp_call", "bp", "fs_cg", "bpcg"):
        imgs, ang, half = _bp_inputs(nx, n, rng, seed)
        inplane = np.stack([rng.uniform(-180, 180, n), rng.uniform(-3, 3, n), rng.uniform(-3, 3, n)], 1)
        return {"imgs": imgs, "ang": ang, "half": half, "inplane": inplane.astype(np.float32)}
    ang = _angles(n, rng)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed + 1)
    if k == "fs_grad":
        N = 2 * nx
        grid = torch.randn((N, N, nx + 1, 2), device=DEV, generator=gen)
        return {"ang": ang, "grid": grid, "g": torch.randn((n, N, nx + 1, 2), device=DEV, generator=gen)}
    s = {"ang": ang, "vol": _volume(nx, _blobs(nx, rng), seed)}
    if k == "pj3q_grad":
        s["g"] = torch.randn((n, nx, nx), device=DEV, generator=gen)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    k = case["kind"]
    if k == "multi":
        s["ctxs"] = [ops.Context(0) for _ in s["classes"]]
        return s
    s["ctx"] = ops.Context(0)
    if k == "bp" and case["host"]:
        s["imgs"] = torch.empty(s["imgs"].shape, pin_memory=True).copy_(s["imgs"]).numpy()
    if k == "bpcg":
        s["imgs"] = s["imgs"].cpu().numpy()
    if k == "pj3q_grad":
        s["vol"].requires_grad_(True)
    if k in ("fs_grad", "fs_cg"):
        s["plan"] = ag.FourierSlicePlan(case["nx"], s["ang"], ctx=s["ctx"])
    if k == "fs_grad":
        s["grid"].requires_grad_(True)
    if k == "fs_cg":
        s["solver"] = ag.NormalCG(s["plan"], 1e-3, case["iters"])
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "bp_call":
        return ops.bp3f(s["imgs"], s["ang"], ctx=s["ctx"], device_out=True)
    if k == "bp":
        ctx = s["ctx"]   # stays open between reconstructions of one box size: grids, buffers and plans are kept
        ctx.bp_open(case["nx"], case["grids"], _sym(case["sym"]), bf16=case["bf16"])
        ctx.bp_insert(s["imgs"], s["ang"], s["half"] if case["grids"] == 2 else None,
                      inplane=s["inplane"] if case["inplane"] else None)
        return ctx.bp_finish(("all", "1", "2") if case["grids"] == 2 else ("all",), device=True)
    if k == "multi":
        return ops.bp32f_multiclass(s["classes"], ctxs=s["ctxs"], device_out=True)
    if k == "pj3q":
        return ops.pj3q(s["vol"], s["ang"], ctx=s["ctx"])
    if k == "pj3q_grad":
        p = ag.pj3q(s["vol"], s["ang"], ctx=s["ctx"])
        (g,) = torch.autograd.grad(p, s["vol"], s["g"])
        return {"proj": p.detach(), "grad": g}
    if k == "pj3f":
        return ops.pj3f(s["vol"], s["ang"], ctx=s["ctx"])
    if k == "fs_grad":
        t = ag.fourier_slice(s["grid"], s["plan"])
        (g,) = torch.autograd.grad(t, s["grid"], s["g"])
        return {"slices": t.detach(), "grad": g}
    if k == "fs_cg":
        x = ag.cg_reconstruct(s["plan"].stage(s["imgs"]), s["solver"])
        return {"grid": x, "vol": s["plan"].volume(x)}
    vol, log = ops.bpcg(s["imgs"], s["ang"], errm=1e-9, maxit=case["iters"], lam=1e-3, ctx=s["ctx"])
    return {"vol": vol, "log": log}


# ---------------------------------------------------------------------------- work
def work(case):
    k = case["kind"]
    if k == "multi":
        boxes = [int(b) for b in case["boxes"].split(",")]
        each = [work({"kind": "bp", "nx": b, "images": case["images"] / len(boxes), "grids": 2, "sym": 1})
                for b in boxes]
        return {q: sum(w[q] for w in each) for q in ("bytes", "flops")}
    nx, n = case["nx"], case["images"]
    N, vol, img = 2 * nx, 4.0 * nx ** 3, 4.0 * nx ** 2
    taps = 0.5 * math.pi * nx ** 2 * 3.6 ** 3 * 0.98   # of one slice
    fft2, fft3 = 2.5 * N * N * 2 * math.log2(N), 2.5 * N ** 3 * 3 * math.log2(N)
    grid = 8.0 * N * N * (nx + 1)
    ball = math.pi / 6 * nx ** 3   # samples of one projection
    if k in ("bp_call", "bp"):
        outs = 3 if case.get("grids", 1) == 2 else 1
        return {"bytes": n * img + outs * vol, "flops": n * (fft2 + case.get("sym", 1) * taps * 8) + outs * fft3}
    if k in ("pj3q", "pj3f"):
        return {"bytes": vol + n * img, "flops": n * ball * (24 if k == "pj3q" else 240)}
    if k == "pj3q_grad":
        return {"bytes": 2 * (vol + n * img), "flops": n * ball * 56}
    if k == "fs_grad":
        return {"bytes": 2 * (grid + n * 8.0 * N * (nx + 1)), "flops": n * taps * 12}
    if k == "fs_cg":
        return {"bytes": n * img + grid + vol, "flops": n * (fft2 + taps * 6 + case["iters"] * taps * 10) + fft3}
    return {"bytes": n * img + vol, "flops": n * ball * 0.9 * (10 + case["iters"] * 22)}


# ---------------------------------------------------------------------------- exact: gridding
def _i1(x):
    t2, term = (0.5 * x) ** 2, 0.5 * x
    out = term
    for k in range(1, 100):
        term = term * t2 / (k * (k + 1.0))
        out = out + term
    return out


def _kb(N):
    """FILLBESSIL's table (REAL), FLTB and AAAA for padded size N."""
    f = np.float32
    n2, alpha = f(N), f(6.5)
    aaaa, fltb = f(0.9) * (f(4) / f(2) / n2), f(4999) / f(3)
    b0 = np.sqrt(alpha) * f(_i1(6.5))
    q = np.arange(5000, dtype=f) / fltb / n2
    inside = q <= aaaa
    r = np.where(inside, q / aaaa, f(1))
    ax = alpha * np.sqrt(f(1) - r * r)
    tab = np.where(inside, np.sqrt(ax) * _i1(ax.astype(np.float64)).astype(f) / b0, f(0))
    return torch.as_tensor(tab.astype(f), device=DEV), float(fltb), float(aaaa)


def _wkb(nx, aaaa):
    """|WKB| of WINDKB2A by squared radius: the transform of the table's function, half-integer Bessel of order 3/2."""
    f = np.float32
    l2 = (nx // 2) ** 2
    t = f(2) * f(math.pi) * f(aaaa)
    sigma = (t * t) * np.arange(l2 + 1, dtype=f) - f(6.5) * f(6.5)
    x = np.sqrt(np.abs(sigma.astype(np.float64))) + 1e-300
    small = x < 0.5
    y = np.where(small, 1.0, x)
    # I_3/2(x)/x^3/2 and J_3/2(x)/x^3/2, both times sqrt(pi/2)
    big = np.where(sigma < 0, (np.cosh(y) - np.sinh(y) / y) / y ** 2, (np.sin(y) / y - np.cos(y)) / y ** 2)
    z = np.where(small, np.where(sigma < 0, 1, -1) * x * x, 0.0)
    ser = (1 + z / 10 * (1 + z / 28 * (1 + z / 54 * (1 + z / 88 * (1 + z / 130))))) / 3
    w = np.abs(np.where(small, ser, big) / ((math.cosh(6.5) - math.sinh(6.5) / 6.5) / 6.5 ** 2))
    w[np.abs(sigma) < 1e-7] = 1.0
    return torch.as_tensor(w.astype(f), device=DEV).double()


def _padded_spectra(imgs):
    """Half spectra [n, N, nx+1] complex128 of the padded images: border mean removed, centre moved to the origin."""
    n, nx = imgs.shape[0], imgs.shape[1]
    N = 2 * nx
    g = torch.arange(nx, device=DEV) - nx // 2
    border = (g[:, None] ** 2 + g[None, :] ** 2) > (nx // 2) ** 2
    x = imgs.double()
    x = x - x[:, border].sum(1)[:, None, None] / float(border.sum())
    ip = (N - nx) // 2 + nx % 2
    pad = torch.zeros((n, N, N), dtype=torch.float64, device=DEV)
    at = (torch.arange(nx, device=DEV) + ip - nx) % N
    pad[:, at[:, None], at[None, :]] = x
    return torch.fft.rfft2(pad)


class _Slices:
    """Pixels and taps of a chunk of central slices: coordinates, table index and weight in REAL (ONELINE)."""

    def __init__(self, nx):
        self.nx, self.N = nx, 2 * nx
        I = torch.arange(0, nx + 1, device=DEV)
        J = torch.arange(-nx + 1, nx + 1, device=DEV)
        jj, ii = torch.meshgrid(J, I, indexing="ij")
        keep = (ii * ii + jj * jj < nx * nx) & ~((ii == 0) & (jj < 0))
        self.I, self.J = ii[keep], jj[keep]
        self.pix = torch.where(self.J >= 0, self.J, self.N + self.J) * (nx + 1) + self.I
        self.tab, self.fltb, self.aaaa = _kb(self.N)

    def place(self, dm):
        """dm [b, 6] float32: coordinates with x >= 0, the flip flag and the first nonzero tap of each axis."""
        nx, N = self.nx, self.N
        fi, fj = self.I.float(), self.J.float()
        v = [fi * dm[:, k:k + 1] + fj * dm[:, k + 3:k + 4] for k in range(3)]
        flip = v[0] < 0
        v = [torch.where(flip, -t, t) for t in v]
        near = [((t + 0.5) + float(N)).to(torch.int32) - N for t in v]
        ok = near[0] <= nx - 3
        for t in near[1:]:
            ok &= (t >= -nx + 4) & (t <= nx - 3)
        first = [t - 2 + (self._w(c, t - 2) == 0).int() for c, t in zip(v, near)]
        return v, flip, ok, first

    def _w(self, c, k):
        d = (c - k.float()).abs() * self.fltb
        f = d.floor()
        return self.tab[(f.int() + (d - f >= 0.5).int()).clamp(max=4999)]

    def taps(self, dm):
        """Yields (voxel index, weight, reflected) of the 64 taps of every pixel; weight 0 where there is none."""
        nx, N = self.nx, self.N
        v, flip, ok, first = self.place(dm)
        w = [[self._w(c, f + l) for l in range(4)] for c, f in zip(v, first)]
        for lx in range(4):
            x = first[0] + lx
            refl = x < 0
            for lz in range(4):
                z = first[2] + lz
                z = torch.where(refl, -z, z) % N
                for ly in range(4):
                    y = first[1] + ly
                    y = torch.where(refl, -y, y) % N
                    wg = (w[0][lx] * (w[1][ly] * w[2][lz])) * ok
                    yield (z.long() * N + y) * (nx + 1) + x.abs().clamp(max=nx), wg.double(), refl
        self.flip = flip


def _chunks(n, nx):
    b = max(1, int(4e6 / (1.6 * nx * nx)))
    return [(a, min(n, a + b)) for a in range(0, n, b)]


def _add_slices(sl, dm, btq, X, W=None):
    """X += BTQ w (conjugate at reflected taps), W += w for one chunk; btq [b, pixels] complex128 already flipped."""
    for idx, wg, refl in sl.taps(dm):
        idx = idx.reshape(-1)
        X[0].index_add_(0, idx, (btq.real * wg).reshape(-1))
        X[1].index_add_(0, idx, (torch.where(refl, -btq.imag, btq.imag) * wg).reshape(-1))
        if W is not None:
            W.index_add_(0, idx, wg.reshape(-1))


def _exact_bp(imgs, ang, half, nx, grids, sym, bf16=False):
    N = 2 * nx
    sl = _Slices(nx)
    X = [torch.zeros((2, N * N * (nx + 1)), dtype=torch.float64, device=DEV) for _ in range(grids)]
    W = [torch.zeros(N * N * (nx + 1), dtype=torch.float64, device=DEV) for _ in range(grids)]
    dms = _cang(ang)
    rot = [None] if sym is None else list(_cang(sym))
    for g in range(grids):
        mine = np.arange(len(ang)) if grids == 1 else np.flatnonzero((half == 0) == g)
        for a, b in _chunks(len(mine), nx):
            at = mine[a:b]
            sp = _padded_spectra(imgs[torch.as_tensor(at, device=DEV)]).reshape(len(at), -1)[:, sl.pix]
            if bf16:
                sp = torch.complex(sp.real.float().bfloat16().double(), sp.imag.float().bfloat16().double())
            for r in rot:
                d = dms[at]
                if r is not None:   # MATMUL in REAL, the sum in order
                    m = d.reshape(-1, 3, 3)
                    d = np.stack([(r[i] * m[:, j, 0] + r[i + 3] * m[:, j, 1]) + r[i + 6] * m[:, j, 2]
                                  for j in range(3) for i in range(3)], 1)
                d = torch.as_tensor(d[:, :6], device=DEV)
                flip = sl.place(d)[1]
                _add_slices(sl, d, torch.where(flip, sp, sp.conj()), X[g], W[g])
    V = []
    for g in range(grids):
        Xc = torch.complex(X[g][0], X[g][1]).reshape(N, N, nx + 1)
        Wc = W[g].reshape(N, N, nx + 1)
        m = (-torch.arange(N, device=DEV)) % N
        p, q = Xc[:, :, 0].clone(), Wc[:, :, 0].clone()
        p2, q2 = p + p[m][:, m].conj(), q + q[m][:, m]
        keep = torch.zeros((N, N), dtype=torch.bool, device=DEV)   # the origin and the Nyquist lines stay
        keep[nx, :] = keep[:, nx] = keep[0, 0] = True
        Xc[:, :, 0], Wc[:, :, 0] = torch.where(keep, p, p2), torch.where(keep, q, q2)
        V.append((Xc, Wc))
    if grids == 1:
        return _finish(V[0][0], V[0][1], nx, sl.aaaa, sym)
    return {"all": _finish(V[0][0] + V[1][0], V[0][1] + V[1][1], nx, sl.aaaa, sym),
            "1": _finish(*V[0], nx, sl.aaaa, sym), "2": _finish(*V[1], nx, sl.aaaa, sym)}


def _radius2(nx):
    g = torch.arange(nx, device=DEV) - nx // 2
    return g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2


def _crop(F, nx):
    """Inverse transform of a grid (SPIDER's sign and phase), centred nx^3."""
    N = 2 * nx
    k, i = torch.arange(N, device=DEV), torch.arange(nx + 1, device=DEV)
    s = 1.0 - 2.0 * ((k[:, None, None] + k[None, :, None] + i[None, None, :]) % 2)
    F = (F * s).conj().resolve_conj()
    F[0, 0, 0] = F[0, 0, 0].real.clone()
    ip = (N - nx) // 2 + nx % 2
    return torch.fft.irfftn(F, s=(N, N, N))[ip:ip + nx, ip:ip + nx, ip:ip + nx]


def _finish(X, W, nx, aaaa, sym):
    X = torch.where(W > 0.1, X / W.clamp(min=1e-30), torch.zeros_like(X))
    r2, l2 = _radius2(nx), (nx // 2) ** 2
    wkb = _wkb(nx, aaaa)
    v = _crop(X, nx) / wkb[r2.clamp(max=l2)]
    shell = (r2 >= (nx // 2 - 1) ** 2) & (r2 <= l2)
    v = torch.where(r2 <= l2, v - v[shell].sum() / float(shell.sum()), torch.zeros_like(v))
    return v if sym is None else _symvol(v, nx, _cang(sym))


def _symvol(v, nx, rot):
    lo = -(nx // 2)
    hi = nx // 2 - 1 if nx % 2 == 0 else nx // 2
    g = torch.arange(nx, device=DEV, dtype=torch.float64) + lo
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    inside = (x * x + y * y + z * z) <= (min(abs(lo), abs(hi)) - 1) ** 2
    x, y, z = x[inside], y[inside], z[inside]
    out, flat = torch.zeros_like(v), v.reshape(-1)
    for R in rot.astype(np.float64):
        t = v.clone()
        if not (R[0] == R[4] == R[8] == 1.0):
            p = [R[3 * k] * x + R[3 * k + 1] * y + R[3 * k + 2] * z for k in range(3)]
            f = [q.floor() for q in p]
            d = [q - h for q, h in zip(p, f)]
            L = [[q * (q - 1) / 2, 1 - q * q, q * (q + 1) / 2] for q in d]
            f = [h.long() - lo for h in f]
            s = 0.0
            for c in range(3):
                for b in range(3):
                    for a in range(3):
                        at = ((f[2] + c - 1) * nx + (f[1] + b - 1)) * nx + (f[0] + a - 1)
                        s = s + flat[at] * L[0][a] * L[1][b] * L[2][c]
            t[inside] = s
        out += t
    return out


def _rtsq(imgs, prm):
    """RTSQ: each image rotated and shifted by quadratic interpolation with wrapped indices (QUADRI).  The quadratics
    of neighbouring cells do not join, so the coordinates, which choose the cell, are REAL; the sums are 64-bit."""
    n, nx = imgs.shape[0], imgs.shape[1]
    out = torch.empty(imgs.shape, dtype=torch.float64, device=DEV)
    cen = nx // 2 + 1
    r1, r2 = float(-(nx // 2)), float(nx // 2 - 1 if nx % 2 == 0 else nx // 2)
    wrap = float(nx if nx % 2 == 0 else nx + 1)
    g = torch.arange(1, nx + 1, device=DEV, dtype=torch.float32)
    dgr = np.float32(math.pi) / np.float32(180)
    for b in range(n):
        th = np.float32(prm[b, 0]) * dgr
        co, si = float(np.cos(th)), float(np.sin(th))
        t = []
        for k in (1, 2):
            q = g + float(np.float32(-cen) - np.float32(math.fmod(float(prm[b, k]), nx)))
            q = torch.where(q < r1, (q + wrap).clamp(max=r2), q)
            t.append(torch.where(q > r2, (q - wrap).clamp(min=r1), q))
        xi, yi = t[0][None, :], t[1][:, None]
        x, y = xi * co + (-yi * si + cen), xi * si + (yi * co + cen)
        p = []
        for q in (x, y):
            q = torch.where(q < 1, q + (1 - torch.trunc(q / nx)) * nx, q)
            p.append(torch.where(q > nx + 0.5, torch.fmod(q - 1, nx) + 1, q))
        i, j = p[0].long(), p[1].long()
        dx, dy = (p[0] - i).double(), (p[1] - j).double()
        f = imgs[b].double()

        def at(a, c):
            return f[(c - 1) % nx, (a - 1) % nx]
        f0 = at(i, j)
        c1, c3 = at(i + 1, j) - f0, at(i, j + 1) - f0
        c2, c4 = (c1 - f0 + at(i - 1, j)) / 2, (c3 - f0 + at(i, j - 1)) / 2
        c5 = at(i + 1, j + 1) - f0 - c1 - c3   # coordinates are positive, so HXC = HYC = 1
        out[b] = f0 + dx * (c1 + (dx - 1) * c2 + dy * c5) + dy * (c3 + (dy - 1) * c4)
    return out


# ---------------------------------------------------------------------------- exact: projectors
def _ball(nx, ri):
    """Centred coordinates (x, y, z) of the voxels inside radius ri and their output pixel."""
    g = torch.arange(nx, device=DEV, dtype=torch.float64) - nx // 2
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    m = x * x + y * y + z * z <= ri * ri
    x, y, z = x[m], y[m], z[m]
    return x, y, z, (y.long() + nx // 2) * nx + x.long() + nx // 2


def _trilinear(nx, dm, x, y, z):
    """Corner indices and weights of the sample positions of one projection (weight 0 outside the volume)."""
    p = [x * dm[k] + y * dm[k + 3] + z * dm[k + 6] + (nx // 2 + 1) for k in range(3)]
    i = [torch.trunc(q) for q in p]
    ok = torch.ones_like(x, dtype=torch.bool)
    for q in i:
        ok &= (q >= 1) & (q < nx)
    d = [q - h for q, h in zip(p, i)]
    i = [torch.where(ok, h, torch.ones_like(h)).long() for h in i]
    base = ((i[2] - 1) * nx + (i[1] - 1)) * nx + i[0] - 1
    for c in (0, 1):
        for b in (0, 1):
            wyz = (d[2] if c else 1 - d[2]) * (d[1] if b else 1 - d[1]) * ok
            for a in (0, 1):
                yield base + (c * nx + b) * nx + a, wyz * (d[0] if a else 1 - d[0])


def _exact_pj3q(vol, ang, g=None):
    nx = vol.shape[0]
    x, y, z, pix = _ball(nx, float(nx // 2 - 2))
    flat = vol.detach().double().reshape(-1)
    out = torch.zeros((len(ang), nx * nx), dtype=torch.float64, device=DEV)
    grad = None if g is None else torch.zeros_like(flat)
    for a, dm in enumerate(_cang(ang).astype(np.float64)):
        s = 0.0
        gp = None if g is None else g[a].double().reshape(-1)[pix]
        for at, w in _trilinear(nx, dm, x, y, z):
            s = s + flat[at] * w
            if gp is not None:
                grad.index_add_(0, at, gp * w)
        out[a].index_add_(0, pix, s)
    out = out.reshape(-1, nx, nx)
    return out if g is None else {"proj": out, "grad": grad.reshape(vol.shape)}


def _fbs3(vol):
    """Value and derivative tables {F, X, Y, XY, Z, XZ, YZ, XYZ} of FBS3_PREP by Fourier derivatives."""
    n = vol.shape[0]
    a4 = np.float32(6.28318530717958647692) / np.float32(n)

    def freq(m):
        k = np.arange(m)
        k = np.where(k <= n // 2, k, k - n).astype(np.float32)
        return torch.as_tensor((k * a4).astype(np.float64), device=DEV)
    w, h = freq(n), n // 2 + 1
    if n % 2 == 0:
        w[n // 2] = 0
    wx, wy, wz = freq(n)[None, None, :h], w[None, :, None], w[:, None, None]
    F = torch.fft.rfftn(vol.double()).conj().resolve_conj()
    x1, y1 = -1j * wx * F, -1j * wy * F
    xy = -1j * wy * x1
    # the table's XZ takes X's real part for both components
    spec = [x1, y1, xy, -1j * wz * F, torch.complex(x1.real * wz, -x1.real * wz), -1j * wz * y1, -1j * wz * xy]
    m = (-torch.arange(n, device=DEV)) % n
    out = [vol.double()]
    for G in spec:
        for c in {0, n // 2} if n % 2 == 0 else {0}:   # Hermitian part, what a real inverse keeps
            G[:, :, c] = (G[:, :, c] + G[:, :, c][m][:, m].conj()) / 2
        out.append(torch.fft.irfftn(G.conj().resolve_conj(), s=(n, n, n)))
    return [t.reshape(-1) for t in out]


def _cub(f0, d0, f1, d1, t):
    a2, a3 = 3 * (f1 - f0) - 2 * d0 - d1, 2 * (f0 - f1) + d0 + d1
    return f0 + t * (d0 + t * (a2 + t * a3))


def _exact_pj3f(vol, ang):
    nx = vol.shape[0]
    T = torch.stack(_fbs3(vol), 1)
    x, y, z, pix = _ball(nx, float(nx // 2 - 2))
    out = torch.zeros((len(ang), nx * nx), dtype=torch.float64, device=DEV)
    for a, dm in enumerate(_cang(ang).astype(np.float64)):
        p = [x * dm[k] + y * dm[k + 3] + z * dm[k + 6] + (nx // 2 + 1) for k in range(3)]
        i = [q.floor() for q in p]
        d = [q - h for q, h in zip(p, i)]
        i = [(h.long() - 1) % nx for h in i]
        j = [(h + 1) % nx for h in i]
        pl = []
        for zz in (i[2], j[2]):
            q00, q10, q01, q11 = (T[(zz * nx + yy) * nx + xx] for yy in (i[1], j[1]) for xx in (i[0], j[0]))
            for o in (0, 4):   # the value plane and its z derivative
                u = [_cub(l[:, o + c], l[:, o + c + 1], r[:, o + c], r[:, o + c + 1], d[0])
                     for l, r, c in ((q00, q10, 0), (q00, q10, 2), (q01, q11, 0), (q01, q11, 2))]
                pl.append(_cub(u[0], u[1], u[2], u[3], d[1]))
        out[a].index_add_(0, pix, _cub(pl[0], pl[1], pl[2], pl[3], d[2]))
    return out.reshape(-1, nx, nx)


# ---------------------------------------------------------------------------- exact: central slices and CG
def _extract(sl, dm, X):
    acc = [0.0, 0.0]
    for idx, wg, refl in sl.taps(dm):
        acc[0] = acc[0] + X[0][idx] * wg
        acc[1] = acc[1] + torch.where(refl, -X[1][idx], X[1][idx]) * wg
    t = torch.complex(*acc)
    return torch.where(sl.flip, t, t.conj())   # the slice value


def _planes(grid):
    return torch.stack([grid[..., 0].detach().double().reshape(-1), grid[..., 1].detach().double().reshape(-1)])


def _exact_fs_grad(grid, ang, g, nx):
    N = 2 * nx
    sl, X = _Slices(nx), _planes(grid)
    dms = torch.as_tensor(_cang(ang)[:, :6], device=DEV)
    out = torch.zeros((len(ang), N * (nx + 1), 2), dtype=torch.float64, device=DEV)
    G = torch.zeros_like(X)
    for a, b in _chunks(len(ang), nx):
        out[a:b, sl.pix] = torch.view_as_real(_extract(sl, dms[a:b], X).resolve_conj())
        t = torch.view_as_complex(g[a:b].double().reshape(b - a, -1, 2).contiguous())[:, sl.pix]
        _add_slices(sl, dms[a:b], torch.where(sl.flip, t, t.conj()), G)
    return {"slices": out.reshape(len(ang), N, nx + 1, 2), "grad": G.T.reshape(N, N, nx + 1, 2)}


def _exact_fs_cg(imgs, ang, nx, iters, lam):
    N = 2 * nx
    sl = _Slices(nx)
    dms = torch.as_tensor(_cang(ang)[:, :6], device=DEV)
    r = torch.zeros((2, N * N * (nx + 1)), dtype=torch.float64, device=DEV)
    for a, b in _chunks(len(ang), nx):
        t = _padded_spectra(imgs[a:b]).reshape(b - a, -1)[:, sl.pix]
        _add_slices(sl, dms[a:b], torch.where(sl.place(dms[a:b])[1], t, t.conj()), r)
    x, p = torch.zeros_like(r), r.clone()
    rs = (r * r).sum()
    for _ in range(iters):
        ap = lam * p
        for a, b in _chunks(len(ang), nx):
            t = _extract(sl, dms[a:b], p)
            _add_slices(sl, dms[a:b], torch.where(sl.flip, t, t.conj()), ap)
        alpha = rs / (p * ap).sum()
        x, r = x + alpha * p, r - alpha * ap
        new = (r * r).sum()
        p, rs = r + (new / rs) * p, new
    X = torch.complex(x[0], x[1]).reshape(N, N, nx + 1)
    grid = torch.view_as_real(X).clone()
    m = (-torch.arange(N, device=DEV)) % N
    X[:, :, 0] = (X[:, :, 0] + X[:, :, 0][m][:, m].conj()) / 2
    r2, l2 = _radius2(nx), (nx // 2) ** 2
    v = _crop(X, nx) * _wkb(nx, sl.aaaa)[r2.clamp(max=l2)]
    return {"grid": grid, "vol": torch.where(r2 <= l2, v, torch.zeros_like(v))}


def _fixedge(p):
    """FIXEDGE, mode 1: the first and last nonzero of every line extended by one voxel, along x, y, then z."""
    n = p.shape[0]
    for ax in (2, 1, 0):
        q = p.movedim(ax, -1).clone()
        nz = q != 0
        any_ = nz.any(-1)
        f = nz.to(torch.int8).argmax(-1)
        l = n - 1 - nz.flip(-1).to(torch.int8).argmax(-1)
        for at, step in ((f, -1), (l, 1)):
            to = at + step
            ok = any_ & (to >= 0) & (to < n)
            v = q.gather(-1, at[..., None])[..., 0]
            to = to.clamp(0, n - 1)[..., None]
            q.scatter_(-1, to, torch.where(ok, v, q.gather(-1, to)[..., 0])[..., None])
        p = q.movedim(-1, ax)
    return p.contiguous()


def _exact_bpcg(imgs, ang, nx, iters, lam):
    imgs = torch.as_tensor(imgs, device=DEV).double()
    n, ri, ldp = len(ang), float(nx // 2 - 2), nx // 2 + 1
    g = torch.arange(nx, device=DEV, dtype=torch.float64) - nx // 2
    zz, yy, xx = torch.meshgrid(g, g, g, indexing="ij")
    m = xx * xx + yy * yy + zz * zz <= ri * ri
    x, y, z = xx[m], yy[m], zz[m]

    def bilinear(dm):
        px, py = x * dm[0] + y * dm[1] + z * dm[2] + ldp, x * dm[3] + y * dm[4] + z * dm[5] + ldp
        i, j = px.trunc(), py.trunc()
        dx, dy = px - i, py - j
        at = ((j - 1) * nx + i - 1).long()
        return [(at, (1 - dx) * (1 - dy)), (at + 1, dx * (1 - dy)), (at + nx, (1 - dx) * dy), (at + nx + 1, dx * dy)]
    cb = torch.zeros_like(x)
    for k, dm in enumerate(_cang(ang).astype(np.float64)):
        f = imgs[k].reshape(-1)
        for at, w in bilinear(dm):
            cb += f[at] * w
    circ = (g[:, None] ** 2 + g[None, :] ** 2) <= ri * ri
    aba = imgs[:, ~circ].sum() / (float((~circ).sum()) * n)
    kls = float(circ.sum()) * n
    cb -= aba * n
    inside = imgs[:, circ]
    chi2 = (inside ** 2).sum() - aba * (2 * inside.sum() - aba * kls)
    bnorm = (cb * cb).sum()
    # HIANG: theta folded to below 90, phi cut to 0.01 degree, psi dropped (all REAL)
    th, ph = ang[:, 1].copy(), ang[:, 2].copy()
    fold = th >= 90
    th[fold] = np.float32(180) - th[fold]
    ph[fold] = ph[fold] + np.float32(180)
    ph[fold & (ph >= 360)] -= np.float32(360)
    ph = (np.float32(100) * ph).astype(np.int32).astype(np.float32) / np.float32(100)
    dms = _cang(np.stack([np.zeros_like(ph), th, ph], 1)).astype(np.float64)
    sol, p, q, log = torch.zeros_like(x), torch.zeros_like(x), 0.0, []
    for it in range(iters):
        delsq = (cb * cb).sum()
        p = cb - q * delsq * p
        q = -1.0 / delsq
        e = torch.zeros_like(x)
        for dm in dms:
            taps = bilinear(dm)
            im = torch.zeros(nx * nx, dtype=torch.float64, device=DEV)
            for at, w in taps:
                im.index_add_(0, at, p * w)
            for at, w in taps:
                e += im[at] * w
        P = torch.zeros((nx, nx, nx), dtype=torch.float64, device=DEV)
        P[m] = p
        P = _fixedge(P)
        lap = 6 * P
        for ax in range(3):
            lap = lap - P.roll(1, ax) - P.roll(-1, ax)
        e += float(np.float32(lam)) * lap[m]
        step = delsq / (p * e).sum()
        chi2 = chi2 - step * delsq
        log.append([float(it + 1), float(delsq / bnorm), float(chi2)])
        sol, cb = sol + step * p, cb - step * e
    v = torch.zeros((nx, nx, nx), dtype=torch.float64, device=DEV)
    v[m] = sol
    return {"vol": v, "log": torch.tensor(log, dtype=torch.float64)}


def exact(case, seed):
    s = _inputs(case, seed)
    k = case["kind"]
    if k == "multi":
        out = []
        for imgs, ang, half in s["classes"]:
            o = _exact_bp(imgs, ang, half, imgs.shape[1], 2, None)
            out.append((o["all"], o["1"], o["2"]))
        return out
    nx = case["nx"]
    if k == "bp_call":
        return _exact_bp(s["imgs"], s["ang"], s["half"], nx, 1, None)
    if k == "bp":
        imgs = _rtsq(s["imgs"], s["inplane"]) if case["inplane"] else s["imgs"]
        o = _exact_bp(imgs, s["ang"], s["half"], nx, case["grids"], _sym(case["sym"]), case["bf16"])
        return o if case["grids"] == 2 else {"all": o}
    if k == "pj3q":
        return _exact_pj3q(s["vol"], s["ang"])
    if k == "pj3q_grad":
        return _exact_pj3q(s["vol"], s["ang"], s["g"])
    if k == "pj3f":
        return _exact_pj3f(s["vol"], s["ang"])
    if k == "fs_grad":
        return _exact_fs_grad(s["grid"], s["ang"], s["g"], nx)
    if k == "fs_cg":
        return _exact_fs_cg(s["imgs"], s["ang"], nx, case["iters"], 1e-3)
    return _exact_bpcg(s["imgs"], s["ang"], nx, case["iters"], 1e-3)
