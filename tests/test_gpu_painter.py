"""The painter form's second pass: unions within and beyond the intervals that wait for the offsets,
columns beyond the working list, and sizes on both sides of the line where four threads share a column.
The union is of the oracle's own FP64 candidates, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plates", [1, 15, 16, 17, 31, 32, 33, 70])
@pytest.mark.parametrize("r", [0.4, 1.0, 3.7])
def test_painter_unions_of_any_size(ctx, vo, oracle, plates, r):
    """Plates 20 apart: a column's union has as many intervals, one or none of them in every eleventh."""
    nx, ny = 37, 9
    base = 10.0 + 20.0 * np.arange(plates)
    cols = [np.stack([base + 0.1 * (x % 5), base + 1 + 0.3 * (y % 3)], 1) for y in range(ny) for x in range(nx)]
    for c in range(0, nx * ny, 11):
        cols[c] = cols[c][: c % 2]
    offs = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 20.0 * plates + 20), 1.0, 0)
    check(ctx, oracle, grid, offs, np.concatenate(cols).reshape(-1), "dilation", r)


@pytest.mark.parametrize("nx,ny,r", [(1, 1, 2.0), (7, 5, 4.0), (33, 4, 9.5), (255, 257, 1.0), (257, 257, 1.0)])
def test_painter_thread_split(ctx, vo, oracle, nx, ny, r):
    grid, offs, z = vo.synth_volume(vo.SynthSpec(nx, ny=ny, n_spheres=25, s_rmin=1, s_rmax=max(nx, ny) / 6 + 1, n_cyl=4, seed=nx))
    for op in ("dilation", "erosion"):
        check(ctx, oracle, grid, offs, z, op, r)


def check(ctx, oracle, grid, offs, z, op, r):
    v = ctx.upload(grid, offs, np.ascontiguousarray(z, dtype=np.float64))
    out, _ = ctx.morph(v, op, r, "separable")
    assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, r, op), tol=0.0, what=f"{op} r={r}")
    out.free()
    v.free()
