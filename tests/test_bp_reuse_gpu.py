"""Reconstructions that reuse a context's grids: buffers kept over bp_close and
same-size bp_open, partial grids exchanged with the grid by the first fold,
grids left half done.  Each result equals a fresh context's to the order of
the FP32 sums (2e-6)."""
import numpy as np
import pytest

from spider_b200 import ops, synth

pytestmark = pytest.mark.gpu
NX, N = 24, 90


@pytest.mark.parametrize("fold_every", [0, 16])
@pytest.mark.parametrize("end", ["finish", "insert", "flush", "partial", "close"])
def test_reconstruction_after_another(end, fold_every):
    """The first reconstruction ends finished and closed, finished only, after an
    insertion without a finish, flushed, or merged with a partial; with
    one or two grids before and after; folds never, or within the images."""
    rng = np.random.default_rng(7)
    imgs = rng.standard_normal((2, N, NX, NX)).astype(np.float32)
    ang = [synth.so3_angles(N, rng) for _ in range(2)]
    half = synth.half_mask(N, rng)

    def run(c, k, grids):
        c.bp_open(NX, grids)
        c.bp_insert(imgs[k][:50], ang[k][:50], half[:50] if grids == 2 else None)
        c.bp_insert(imgs[k][50:], ang[k][50:], half[50:] if grids == 2 else None)
        return c.bp_finish(("all", "1", "2") if grids == 2 else ("all",))

    def fresh(k, grids):
        c = ops.Context(0)
        try:
            c.set_accumulation(True, fold_every)
            return run(c, k, grids)
        finally:
            c.close()
    c = ops.Context(0)
    try:
        c.set_accumulation(True, fold_every)
        for first, second in ((1, 1), (2, 1), (1, 2), (2, 2)):
            if end in ("finish", "close"):
                run(c, 0, first)
                if end == "close":
                    c.bp_close()
            else:
                c.bp_open(NX, first)
                if end == "partial":
                    x = rng.standard_normal((2 * NX, 2 * NX, NX + 1, 2)).astype(np.float32)
                    c.bp_partial_add(x, np.ones(x.shape[:3], np.float32))
                else:
                    c.bp_insert(imgs[0], ang[0], half if first == 2 else None)
                    if end == "flush":
                        c.bp_flush()
                        c.bp_insert(imgs[0][:20], ang[0][:20], half[:20] if first == 2 else None)
            got, ref = run(c, 1, second), fresh(1, second)
            for k, v in ref.items():
                assert synth.rel_l2(got[k], v) <= 2e-6, (first, second, k)
    finally:
        c.close()


@pytest.mark.parametrize("nx", [24, 147])
def test_calls_of_many_sizes(nx):
    """Calls of seven sizes in turn, each with its own transform batch: the result is that
    of one call of all images, and the plans share one work area, so that after the
    largest call the others take no more device memory."""
    import torch
    sizes = (7, 20, 30, 45, 60, 90, 120)
    m = sum(sizes)
    rng = np.random.default_rng(nx)
    imgs = rng.standard_normal((m, nx, nx)).astype(np.float32)
    ang = synth.so3_angles(m, rng)
    c, one = ops.Context(0), ops.Context(0)
    try:
        one.bp_open(nx, 1)
        one.bp_insert(imgs, ang)
        ref = one.bp_finish(("all",))["all"]
        for turn in range(2):
            c.bp_open(nx, 1)
            end, free = m, []
            for s in sorted(sizes, reverse=True):
                c.bp_insert(imgs[end - s:end], ang[end - s:end])
                end -= s
                free.append(torch.cuda.mem_get_info()[0])
            assert turn == 0 or len(set(free)) == 1
            if turn == 0:
                assert free[0] - free[-1] < 2 << 20   # the plans' constants, no work areas
            assert synth.rel_l2(c.bp_finish(("all",))["all"], ref) <= 2e-6
    finally:
        c.close()
        one.close()


@pytest.mark.parametrize("nx,images,kept", [(64, 200, True), (83, 1100, False), (128, 200, False)])
def test_close_keeps_at_most_its_limit(nx, images, kept):
    """A closed reconstruction leaves at most 512 MB with its context: at 64^3 it stays
    whole; 1,100 images at 83^3 stay below with their buffers but not with the
    transforms' work area (166 = 2 x 83 takes one), 200 at 128^3 with neither."""
    rng = np.random.default_rng(nx)
    imgs = rng.standard_normal((images, nx, nx)).astype(np.float32)
    c = ops.Context(0)
    try:
        empty = c.device_bytes
        c.bp_open(nx, 1)
        c.bp_insert(imgs, synth.so3_angles(images, rng))
        c.bp_finish(("all",))
        full = c.device_bytes
        c.bp_close()
        held = c.device_bytes
        if kept:
            assert held == full <= 512 << 20
        else:
            assert full > 512 << 20 and held - empty < 1 << 20
    finally:
        c.close()
