"""Counts scanned by one block or by many, at the sizes where that changes, and image row reaches passed by
value or tabulated on the device."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (8191, 1), (8192, 1), (8193, 1), (256, 128), (32769, 1), (1, 32768), (3, 21845)])
def test_scan_sizes(ctx, vo, oracle, nx, ny):
    rng = np.random.default_rng(nx + ny)
    n = rng.integers(0, 4, nx * ny)
    n[-1] = 3  # the last column has some
    offs = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    z = np.concatenate([np.sort(rng.choice(200, 2 * k, replace=False)) for k in n]).astype(np.float64) if n.sum() else np.zeros(0)
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 220.0), 1.0, 0)
    v = ctx.upload(grid, offs, z)
    for method in ("fast", "separable"):
        out, _ = ctx.morph(v, "dilation", 1.0, method)
        assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, 1.0, "dilation"), tol=0.0, what=method)
        out.free()
    v.free()


@pytest.mark.parametrize("r", [0.0, 30.9, 31.5, 32.0, 33.2, 70.0])
@pytest.mark.parametrize("h", [1, 20, 45])
def test_image_reach_tables(ctx, oracle, r, h):
    w = 150
    rows = [np.sort(np.random.default_rng(100 * h + i).choice(w, 6, replace=False)) for i in range(h)]
    offs = (6 * np.arange(h + 1)).astype(np.int32)
    ev = np.concatenate(rows).astype(np.int32)
    for op, name in (("dilation", "dilate"), ("erosion", "erode")):
        got, want = ctx.image_morph(w, h, offs, ev, r, op), oracle.image_morph(w, h, offs, ev, r, name)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), op
