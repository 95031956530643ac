"""Dilations by small radii, met column by column: grids on both sides of the line where threads share a
column, grids of one row, radii at the ends of the range, unions beyond the registers and beyond the list
(which go by patches, in a batch by a re-run). The union is of the oracle's own FP64 candidates, so
equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


def check(ctx, oracle, grid, offs, z, op, r):
    z = np.ascontiguousarray(z, dtype=np.float64)
    want = oracle.morph(ogrid(oracle, grid), offs, z, r, op)
    v = ctx.upload(grid, offs, z)
    out, _ = ctx.morph(v, op, r, "fast")
    assert_same(ctx.download(out), want, tol=0.0, what=f"{op} r={r}")
    out.free()
    outs, _ = ctx.morph_batched([v, v], [op, op], [r, r], "fast")
    for o in outs:
        assert_same(ctx.download(o), want, tol=0.0, what=f"batch {op} r={r}")
        o.free()
    v.free()


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 5), (31, 33), (255, 128), (257, 256), (900, 1), (1, 700), (33, 3)])
@pytest.mark.parametrize("r", [0.0, 0.5, 1.0, 2.75, 5.0])
def test_direct_grids(ctx, vo, oracle, nx, ny, r):
    n = max(nx, ny)
    grid, offs, z = vo.synth_volume(vo.SynthSpec(nx, ny=ny, n_spheres=25, s_rmin=1, s_rmax=n / 6 + 1, n_cyl=4, seed=n))
    for op in ("dilation", "erosion"):
        check(ctx, oracle, grid, offs, z, op, r)


@pytest.mark.parametrize("plates", [1, 3, 4, 5, 15, 16, 17, 47, 48, 49, 70])
def test_direct_unions_of_any_size(ctx, vo, oracle, plates):
    """Plates 20 apart: some columns' unions have as many intervals, most columns have none, so that the mean
    stays small."""
    nx, ny = 45, 9
    base = 10.0 + 20.0 * np.arange(plates)
    cols = [np.zeros((0, 2)) for _ in range(nx * ny)]
    for c in range(0, nx * ny, 101):
        cols[c] = np.stack([base + 0.1 * (c % 5), base + 1 + 0.3 * (c % 3)], 1)
    offs = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 20.0 * plates + 20), 1.0, 0)
    for r in (1.0, 3.3):
        check(ctx, oracle, grid, offs, np.concatenate(cols).reshape(-1), "dilation", r)


def test_direct_columns_meet_many_neighbours(ctx, vo, oracle):
    """At most 16 segments per column, all at other heights than the neighbours': 80 intervals in a union."""
    nx, ny = 60, 60
    cols = [np.zeros((0, 2)) for _ in range(nx * ny)]
    for y in range(20, 24):
        for x in range(30, 33):
            base = 10.0 + 50.0 * np.arange(16) + 5.0 * ((x + 3 * y) % 9)
            cols[x + nx * y] = np.stack([base, base + 1], 1)
    offs = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 900.0), 1.0, 0)
    check(ctx, oracle, grid, offs, np.concatenate(cols).reshape(-1), "dilation", 1.0)
