"""The painter form's second pass on columns whose working list is longer on the way than at the end:
groups of segments at other heights in neighbouring columns, and a segment of a farther column that
absorbs one of the groups. Whether the list outgrows its 32 intervals then depends on the order in which
the source columns come, which differs between one thread per column and four."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


def volume(vo, nx, ny, per_group, absorbed):
    """Every six columns along x: four columns of per_group segments, none overlapping another's (the
    third at heights of its own), and one with a segment over the first `absorbed` of the third's."""
    cols = [[] for _ in range(nx * ny)]
    for y in range(ny):
        for x in range(nx):
            k = x % 6
            if k in (0, 1, 3):
                cols[x + nx * y] = [(1000.0 * (1 + k) + 100 * i, 1000.0 * (1 + k) + 100 * i + 1) for i in range(per_group)]
            elif k == 2:
                cols[x + nx * y] = [(5.0 + 8 * i, 6.0 + 8 * i) for i in range(per_group)]
            elif k == 4:
                cols[x + nx * y] = [(0.0, 4.0 + 8 * absorbed)]
    offs = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    z = np.array([v for c in cols for s in c for v in s])
    return vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 6000), 1.0, 0), offs, z


# unions of 17 to 32 intervals that pass 32 on the way; columns on both sides of the line where four threads
# share a column (columns <= 16384 W^2 with W = r + 1: r = 2 up to 147,456)
@pytest.mark.parametrize("nx,ny", [(64, 1), (61, 3), (200, 40), (1536, 100)])
@pytest.mark.parametrize("per_group,absorbed", [(9, 7), (8, 8), (9, 9), (10, 9), (11, 11), (7, 5)])
def test_painter_unions_that_shrink_on_the_way(ctx, vo, oracle, nx, ny, per_group, absorbed):
    grid, offs, z = volume(vo, nx, ny, per_group, absorbed)
    v = ctx.upload(grid, offs, z)
    for op in ("dilation", "erosion"):
        out, _ = ctx.morph(v, op, 2.0, "separable")
        assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, 2.0, op), tol=0.0,
                    what=f"{nx}x{ny} {per_group}/{absorbed} {op}")
        out.free()
    v.free()


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_painter_scattered_segments(ctx, vo, oracle, seed):
    """Segments of a few lengths scattered over the columns: unions from none to beyond 32 intervals."""
    rng = np.random.default_rng(seed)
    nx, ny = 150 + seed, 70
    cols = []
    for _ in range(nx * ny):
        lo = np.sort(rng.uniform(0, 800, rng.poisson(2.2)))
        hi = lo + rng.choice([0.5, 3.0, 60.0], lo.size, p=[0.6, 0.3, 0.1])
        cols.append([(a, min(b, n - 0.25)) for a, b, n in zip(lo, hi, np.append(lo[1:], 2000.0)) if min(b, n - 0.25) > a])
    offs = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    z = np.array([v for c in cols for s in c for v in s])
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 900), 1.0, 0)
    v = ctx.upload(grid, offs, z)
    for r in (2.0, 3.0):
        out, _ = ctx.morph(v, "dilation", r, "separable")
        assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, r, "dilation"), tol=0.0, what=f"r={r}")
        out.free()
    v.free()
