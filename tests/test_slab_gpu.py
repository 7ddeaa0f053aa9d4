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


@pytest.mark.parametrize("nx,nimg", [(8, 9), (15, 40), (16, 1), (17, 40), (33, 60), (40, 700)])
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
