"""The column insertion's and the extraction's geometry on the CPU: every tap of
ONELINE's walk over the pixels is found by exactly one voxel column, from the same
table entries, and nothing is read out of range."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("slab") / "slab_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "slab_check.cpp")],
                   check=True)
    return exe


@pytest.mark.parametrize("nx,count", [(8, 40), (9, 30), (15, 30), (16, 30), (17, 30), (33, 24), (48, 16), (160, 4), (250, 2)])
def test_columns_find_every_tap(check, nx, count):
    """Smallest box, odd boxes, boxes around one and two tiles, large ones; the first
    twelve rotations are the degenerate ones (axes, diagonals, 45 degree planes)."""
    out = subprocess.run([check, str(nx), "5", str(count)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == 2 * count
    for d, banks, cols, nrows, npix, direct, columns, bad in rows:
        assert bad == 0 and direct == columns > 0
        assert nrows <= 47 and npix <= 654
    assert {r[1:3] for r in rows} >= {(2, 2), (2, 1)}
    if count >= 12:
        assert {r[0] for r in rows} == {0, 1, 2}            # every dominant axis
        assert {r[1] for r in rows} == {2, 3}               # shallow and steep slices


@pytest.mark.parametrize("nx,count", [(8, 60), (9, 60), (33, 30), (150, 17), (512, 3)])
def test_extraction_stays_in_range(check, nx, count):
    """Every table entry and voxel of the extraction's windows is in range, and a
    matrix with a NaN or infinite angle or element is not taken for a rotation."""
    out = subprocess.run([check, "extract", str(nx), "7", str(count)], check=True, capture_output=True, text=True).stdout
    assert int(out) == 0
