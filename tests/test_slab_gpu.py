"""The column insertion (insert_x4_kernel) against the oracle's FP64 grids, at
the sizes and orientations where its tiles can go wrong."""
import os

import numpy as np
import pytest

from spider_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _angles(n, seed):
    ang = synth.so3_angles(n, np.random.default_rng(seed))
    # rotations that put the plane on an axis, a diagonal and the x = 0 flip line
    a = float(np.degrees(np.arccos(1 / np.sqrt(3))))
    sp = [(0, 0, 0), (0, 90, 0), (0, 90, 90), (45, 0, 0), (0, 45, 0), (45, a, 45), (0, 180, 0), (90, 90, 45)]
    ang[:len(sp)] = np.array(sp, np.float32)
    return ang


# rows of tiles split into parts (a launch of few slices) and whole ones (1,000 at 33^3)
@pytest.mark.parametrize("nx,nimg", [(8, 9), (15, 40), (16, 1), (17, 40), (33, 60), (33, 1000), (40, 700)])
def test_columns_match_oracle_grids(ctx, orc, nx, nimg):
    """X and W grids within 2e-6 of the FP64 sums: the products' three roundings
    (1e-7) and the random walk of at most a few hundred FP32 additions of 6e-8
    per voxel, plus the FP32 transform's 3e-7."""
    rng = np.random.default_rng(nx)
    imgs = rng.standard_normal((nimg, nx, nx)).astype(np.float32)
    ang = _angles(max(nimg, 8), nx)[:nimg]
    x, w = ops.bp3f_partial(imgs, ang, ctx=ctx)
    xr, wr = orc.bp3f_partial(imgs, ang, prec=1, nthreads=1)
    assert synth.rel_l2(w, wr) <= 2e-6
    assert synth.rel_l2(x, np.stack([xr.real, xr.imag], -1)) <= 2e-6


def _frame(ang):
    """Dominant axis of a slice's normal and the banks of its columns (slab_frame, slab_banks)."""
    psi, th, phi = np.radians(np.asarray(ang, np.float64))
    n = np.array([np.sin(th) * np.cos(phi), np.sin(th) * np.sin(phi), np.cos(th)])
    d = int(np.argmax(np.abs(n)))
    rise = sum(abs(n[a] / n[d]) for a in range(3) if a != d)   # |SU| + |SV|
    return d, 2 if 1.81 * (1 + rise) + 0.01 <= 4.0 else 3


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("banks", [2, 3])
def test_columns_by_frame(ctx, orc, axis, banks, bf16):
    """Slices of one dominant axis and one bank count at a time, FP32 and BF16 spectra:
    W within 2e-6 of the FP64 sums either way; X 2e-6 in FP32, in BF16 2^-9 (half a unit
    of its 8 bits) for every value."""
    nx = 24
    rng = np.random.default_rng(10 * axis + banks)
    ang = synth.so3_angles(900, rng)
    ang = ang[[_frame(a) == (axis, banks) for a in ang]][:40]
    assert len(ang) == 40
    imgs = rng.standard_normal((40, nx, nx)).astype(np.float32)
    ctx.bp_open(nx, 1, bf16=bf16)
    try:
        ctx.bp_insert(imgs, ang)
        x, w = ctx.bp_partial_out(0)
    finally:
        ctx.bp_close()
    xr, wr = orc.bp3f_partial(imgs, ang, prec=1, nthreads=1)
    assert synth.rel_l2(w, wr) <= 2e-6
    assert synth.rel_l2(x, np.stack([xr.real, xr.imag], -1)) <= (2.0 ** -9 if bf16 else 2e-6)


def test_columns_two_classes_in_turn(orc):
    """Classes of two box sizes in one launch, whose tables a CTA loads as it meets
    them: each class's grid is that of its own insertion."""
    rng = np.random.default_rng(31)
    cs = [ops.Context(0), ops.Context(0)]
    try:
        data = []
        for c, nx, n in zip(cs, (20, 33), (300, 200)):
            c.bp_open(nx, 1)
            data.append((rng.standard_normal((n, nx, nx)).astype(np.float32), synth.so3_angles(n, rng)))
        ops.bp_insert_multi(cs, [(imgs, ang, None) for imgs, ang in data])
        for c, (imgs, ang) in zip(cs, data):
            x, w = c.bp_partial_out(0)
            xr, wr = orc.bp3f_partial(imgs, ang, prec=1, nthreads=1)
            assert synth.rel_l2(w, wr) <= 2e-6
            assert synth.rel_l2(x, np.stack([xr.real, xr.imag], -1)) <= 2e-6
    finally:
        for c in cs:
            c.close()


def test_columns_not_finite(ctx):
    """An image with an infinite pixel makes every value of its spectrum infinite
    or NaN: X is then not finite on exactly the voxels that the per-tap
    kernel leaves so, and W is the same."""
    rng = np.random.default_rng(3)
    imgs = rng.standard_normal((6, 24, 24)).astype(np.float32)
    imgs[2, 5, 7] = np.inf
    ang = synth.so3_angles(6, rng)
    x, w = ops.bp3f_partial(imgs, ang, ctx=ctx)
    os.environ["SPI_INSERT"] = "direct"
    try:
        xd, wd = ops.bp3f_partial(imgs, ang, ctx=ctx)
    finally:
        del os.environ["SPI_INSERT"]
    assert np.array_equal(np.isfinite(x), np.isfinite(xd))
    assert not np.isfinite(x).all() and np.isfinite(x).any()
    assert synth.rel_l2(w, wd) <= 1e-6


# few slices go tap by tap, more by columns: from 257 on, FP64 from 41 on at 40^3
@pytest.mark.parametrize("nx,nang", [(8, 3), (15, 20), (16, 1), (17, 20), (40, 300), (40, 41), (8, 300), (15, 300),
                                     (16, 300), (17, 300), (16, 256), (16, 257), (64, 2), (96, 2)])
def test_fourier_slice_pair(ctx, orc, nx, nang):
    """E and E^T at the edges of their tiles and of the routes, FP32 within 2e-6 (as
    above; E sums 64 products) and FP64 within 1e-12 of the oracle pair."""
    import torch

    from spider_b200 import autograd
    rng = np.random.default_rng(100 + nx)
    n = 2 * nx
    ang = _angles(max(nang, 8), nx)[:nang]

    def draw(*shape):
        return rng.standard_normal(shape).astype(np.float32)
    X, T = draw(n, n, nx + 1, 2), draw(nang, n, nx + 1, 2)
    Xc, Tc = (a[..., 0].astype(np.float64) + 1j * a[..., 1] for a in (X, T))
    ref_t, ref_x = orc.fslice_extract(Xc, ang), orc.fslice_insert(Tc, ang)
    ref_n = orc.fslice_insert(ref_t, ang) + 0.25 * Xc

    def off(got, ref):
        g = got.cpu().numpy().astype(np.float64)
        return np.linalg.norm(g[..., 0] + 1j * g[..., 1] - ref) / np.linalg.norm(ref)
    plan = autograd.FourierSlicePlan(nx, ang, ctx=ctx)
    try:
        dX, dT = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
        assert off(plan.forward(dX), ref_t) <= 2e-6
        assert off(plan.adjoint(dT), ref_x) <= 2e-6
        assert off(plan.normal(dX, 0.25), ref_n) <= 4e-6
        assert off(plan.forward64(dX.double()), ref_t) <= 1e-12
        assert off(plan.adjoint64(dT), ref_x) <= 1e-12
        assert off(plan.normal64(dX.double(), 0.25), ref_n) <= 1e-12
    finally:
        plan.close()


def test_fourier_slice_normal_workspaces(ctx):
    """The normal operator through workspaces of one slice, a few and all slices,
    and the entry points without one, give the same; a workspace below
    one slice, misaligned or absent is refused."""
    import ctypes

    import torch

    from spider_b200 import autograd
    nx, nang = 20, 25
    plan = autograd.FourierSlicePlan(nx, _angles(nang, 4), ctx=ctx)
    L, vp, st = plan._L, ctypes.c_void_p, plan._stream()
    try:
        for fp64 in (0, 1):
            dt = torch.float64 if fp64 else torch.float32
            x = torch.randn(plan.shape, dtype=dt, device="cuda")
            per = 2 * nx * (nx + 1) * (16 if fp64 else 8)
            ref = torch.empty_like(x)
            old = L.spi_fslice_normal64 if fp64 else L.spi_fslice_normal
            ops.check(old(plan._h, vp(x.data_ptr()), 0.5, vp(ref.data_ptr()), st))
            ws = torch.empty(nang * (per + 8) + 8, dtype=torch.uint8, device="cuda")
            for slices in (1, 7, nang):
                y = torch.empty_like(x)
                ops.check(L.spi_fslice_normal_ws(plan._h, vp(x.data_ptr()), 0.5, vp(y.data_ptr()), fp64,
                                                 vp(ws.data_ptr()), slices * per + 8 * nang, st))
                assert ((y - ref).norm() / ref.norm()).item() <= (1e-12 if fp64 else 2e-6)
            y = torch.empty_like(x)
            for w, size in ((ws.data_ptr(), per + 8 * nang - 1), (ws.data_ptr() + 8, 2 * per),
                            (None, 2 * per)):
                assert L.spi_fslice_normal_ws(plan._h, vp(x.data_ptr()), 0.5, vp(y.data_ptr()), fp64, vp(w), size,
                                              st) == 101
    finally:
        plan.close()


def test_fourier_slice_normal_without_room(ctx):
    """Where torch cannot give the slice buffer (58 MB), the normal operator runs
    without one, as it did before it had one."""
    import torch

    from spider_b200 import autograd
    nx, nang = 24, 3000
    plan = autograd.FourierSlicePlan(nx, _angles(nang, 8), ctx=ctx)
    try:
        x = torch.randn(plan.shape, dtype=torch.float64, device="cuda")
        ref, got = torch.empty_like(x), torch.empty_like(x)
        plan.normal64(x, 0.5, out=ref)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (1 << 20)) / total)
        try:
            plan.normal64(x, 0.5, out=got)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert ((got - ref).norm() / ref.norm()).item() <= 1e-12
    finally:
        plan.close()


@pytest.mark.parametrize("count", [12, 300])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_fourier_slice_angles_not_finite(ctx, bad, count):
    """A slice with an angle that is not finite has no taps: E writes zeros, E^T and
    the normal operators leave it out, the other slices are as without it."""
    import torch

    from spider_b200 import autograd
    nx = 24
    good = _angles(count, 6)
    ang = np.repeat(good, 2, axis=0)
    for i in range(count):
        ang[2 * i + 1, i % 3] = bad
    X = torch.randn((2 * nx, 2 * nx, nx + 1, 2), device="cuda")
    T = torch.randn((2 * count, 2 * nx, nx + 1, 2), device="cuda")
    plan, ref = autograd.FourierSlicePlan(nx, ang, ctx=ctx), autograd.FourierSlicePlan(nx, good, ctx=ctx)
    try:
        for fwd, x in (("forward", X), ("forward64", X.double())):
            got = getattr(plan, fwd)(x)
            assert torch.equal(got[::2], getattr(ref, fwd)(x))
            assert not got[1::2].any()
        for op, args, rargs, tol in (("adjoint", (T,), (T[::2].contiguous(),), 2e-6),
                                     ("adjoint64", (T,), (T[::2].contiguous(),), 1e-12),
                                     ("normal", (X, 0.25), (X, 0.25), 2e-6),
                                     ("normal64", (X.double(), 0.25), (X.double(), 0.25), 1e-12)):
            got, want = getattr(plan, op)(*args), getattr(ref, op)(*rargs)
            assert ((got - want).norm() / want.norm()).item() <= tol, op
    finally:
        plan.close()
        ref.close()
