"""Segments that a neighbour's candidate holds are passed over: margins at, just below and just above the
growth of H over a step, plates equal over whole areas, and segments wider than any neighbour's. The union is
of the oracle's own FP64 candidates, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


def growths(r):
    """H[d][a - 1] - H[d][a] at a few distances of the disc."""
    d, a = np.meshgrid(np.arange(int(r) + 1), np.arange(1, int(r) + 1), indexing="ij")
    ok = d * d + a * a <= r * r
    h = np.sqrt(r * r - d[ok] ** 2 - (a[ok] - 1) ** 2) - np.sqrt(r * r - d[ok] ** 2 - a[ok] ** 2)
    return np.concatenate([[0.0], h])


@pytest.mark.parametrize("r", [2.0, 5.5, 9.0, 16.0, 31.5])  # the small ones column by column, the others by patches
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_margins_at_the_growth(ctx, vo, oracle, r, seed):
    rng = np.random.default_rng(seed)
    nx, ny = 47, 38
    g = growths(r)
    step = rng.choice(np.concatenate([g, g * (1 + 2**-10), g * (1 - 2**-10), np.nextafter(g, 9.0)]), (ny, nx, 4))
    step *= rng.integers(0, 2, (ny, nx, 4))
    cols = np.empty((ny, nx, 4))
    base = np.array([100.0, 103.0, 180.0, 180.5])
    for y in range(ny):
        for x in range(nx):
            near = cols[y, x - 1] if x else cols[y - 1, x] if y else base
            if rng.random() < 0.05:
                near = base
            cols[y, x] = near + step[y, x] * np.array([-1, 1, -1, 1]) * rng.choice([-1, 1])
            cols[y, x] = np.clip(cols[y, x], [20.0, 101.5, 150.0, 180.25], [101.4, 149.0, 180.2, 300.0])
    offs = (2 * np.arange(nx * ny + 1)).astype(np.int32)
    z = np.ascontiguousarray(cols.reshape(-1))
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 320.0), 1.0, 0)
    v = ctx.upload(grid, offs, z)
    for op in ("dilation", "erosion"):
        out, _ = ctx.morph(v, op, r, "fast")
        assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, r, op), tol=0.0, what=op)
        out.free()
    v.free()
