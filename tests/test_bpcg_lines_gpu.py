"""The mixed-precision BP CG operators (lines of 32 walked together, voxels in
8 x 4 x 4 boxes) against the FP64 operators, at box sizes around their
granules and at view directions along the axes and diagonals, where lines of
a warp project onto one another or onto one image row or column.

Tolerance: a contribution is rounded to half a step of mcap max|x| / (0.95
2^47), mcap = pi (sqrt 2 + sqrt 3 / 2)^2 (2 RI + sqrt 3) bounds the number in a
pixel, so a projection is off by at most mcap^2 2^-48 max|x|, 1.6e-8 at n = 130.
Two CG steps carry the errors of three applications of the operator pair, whose
gain the step lengths undo; with the FP32 rounding of the volume (6e-8) and a
factor of ten for the conditioning, 1e-6 of the largest voxel.  The FP32 tables
("mixed") add 2^-24 for each of the table's four terms and half as much again
for their differences, summed over the images with signs: 4e-6.
"""
import numpy as np
import pytest

from spider_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("mixed64", 1e-6), ("mixed", 4e-6)])
@pytest.mark.parametrize("n,ri,bands", [(8, 2.0, None), (11, 2.0, None), (31, 13.0, None), (33, 14.0, None), (64, 30.0, None),
                                        (66, 30.5, "2"), (66, 31.0, "8"), (130, 62.0, None)])
def test_mixed_operators_match_fp64(ctx, monkeypatch, n, ri, bands, prec, tol):
    if bands:
        monkeypatch.setenv("SPI_CG_BANDS", bands)
    g = np.random.default_rng(n)
    axes = [[0, 0, 0], [0, 90, 0], [0, 90, 90], [0, 45, 0], [0, 45, 90], [0, 90, 45], [0, 54.73, 45], [0, 54.73, 225], [0, 125.26, 135]]
    rest = np.stack([g.uniform(0, 360, 60), np.degrees(np.arccos(g.uniform(-1, 1, 60))), g.uniform(0, 360, 60)], 1)
    ang = np.concatenate([np.array(axes, float), rest]).astype(np.float32)
    x = np.arange(n) - n // 2
    blob = np.exp(-(x[:, None] ** 2 + x[None] ** 2) / (2 * (n / 6.0) ** 2))
    img = (blob + 0.2 * g.standard_normal((len(ang), n, n))).astype(np.float32)
    kw = dict(errm=1e-30, chim=0.0, maxit=2, mode=1, lam=0.5, ctx=ctx)
    v, log = ops.bpcg(img, ang, ri, fp64=prec, **kw)
    ref, rlog = ops.bpcg(img, ang, ri, fp64=True, **kw)
    assert len(log) == len(rlog)
    assert np.abs(ref).max() > 0
    assert np.abs(v - ref).max() <= tol * np.abs(ref).max()


def _solve_case(n, m):
    g = np.random.default_rng(n)
    ang = np.stack([g.uniform(0, 360, m), np.degrees(np.arccos(g.uniform(-1, 1, m))), g.uniform(0, 360, m)], 1).astype(np.float32)
    return g.standard_normal((m, n, n)).astype(np.float32), ang


@pytest.mark.parametrize("n,bands", [(11, None), (33, None), (66, "4"), (130, None)])
def test_projector_without_layouts(ctx, monkeypatch, n, bands):
    """The projector reading the volume itself sums the same integers as from the
    layouts.  The solves' dot products are FP64 sums in any order, 1e-13 of the vectors, and the
    volumes are rounded to FP32: equal to one last bit, 1.2e-7 of the largest voxel."""
    if bands:
        monkeypatch.setenv("SPI_CG_BANDS", bands)
    img, ang = _solve_case(n, 40)
    kw = dict(errm=1e-30, chim=0.0, maxit=2, mode=1, lam=0.5, ctx=ctx, fp64="mixed64")
    ref, _ = ops.bpcg(img, ang, n // 2 - 3.0, **kw)
    monkeypatch.setenv("SPI_CG_LAYOUTS", "0")
    v, _ = ops.bpcg(img, ang, n // 2 - 3.0, **kw)
    assert np.abs(v - ref).max() <= 1.2e-7 * np.abs(ref).max()


def test_solve_without_room_for_layouts():
    """With room for everything but the layouts (268 MB at 256^3), a solve runs without
    them, as it did before it had them."""
    import torch
    n = 256
    img, ang = _solve_case(n, 8)
    kw = dict(errm=1e-30, chim=0.0, maxit=1, mode=1, lam=0.5)
    c = ops.Context(0)
    try:
        ref, _ = ops.bpcg(img, ang, ctx=c, **kw)
        need = c.device_bytes   # with the layouts
    finally:
        c.close()
    c = ops.Context(0)
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - need + (134 << 20), dtype=torch.uint8, device="cuda")
    try:
        v, _ = ops.bpcg(img, ang, ctx=c, **kw)
    finally:
        c.close()
        del fill
        torch.cuda.empty_cache()
    assert np.abs(v - ref).max() <= 1.2e-7 * np.abs(ref).max()


@pytest.mark.parametrize("prec", ["mixed64", "mixed", "fast"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_mixed_angle_not_finite(ctx, bad, prec):
    """A direction with an angle that is not finite is not passed over: the volume is
    NaN where the FP64 operators' is."""
    g = np.random.default_rng(5)
    n, m = 24, 70
    img = g.standard_normal((m, n, n)).astype(np.float32)
    ang = np.stack([g.uniform(0, 360, m), np.degrees(np.arccos(g.uniform(-1, 1, m))), g.uniform(0, 360, m)], 1).astype(np.float32)
    ang[66, 0] = bad   # psi; HIANG takes phi and theta alone, so the merged directions stay finite
    kw = dict(errm=1e-30, chim=0.0, maxit=2, mode=1, lam=0.5, ctx=ctx)
    v, _ = ops.bpcg(img, ang, 9.0, fp64=prec, **kw)
    ref, _ = ops.bpcg(img, ang, 9.0, fp64=True, **kw)
    assert np.isnan(ref).any()
    assert np.array_equal(np.isnan(v), np.isnan(ref))
