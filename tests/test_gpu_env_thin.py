"""The envelope form on long thin grids: its list of line and row segments grows with their number, not with the
square of the longer side (2,000,000 x 1 columns asked for 500 GB). The oracle's own FP64 candidates, so equality
is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2000000, 1), (1, 2000000), (200003, 10), (9, 100001)])
def test_thin_grid(ctx, vo, oracle, nx, ny):
    rng = np.random.default_rng(nx)
    n = nx * ny
    count = np.where(rng.random(n) < 0.02, rng.integers(1, 4, n), 0)
    offs = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
    first = np.repeat(offs[:-1], count)
    lo = 10.0 * (np.arange(offs[-1]) - first) + rng.uniform(1, 3, offs[-1])
    z = np.stack([lo, lo + rng.uniform(0.5, 4, offs[-1])], 1).reshape(-1)
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, 40), 1.0, 0)
    v = ctx.upload(grid, offs, z)
    out, _ = ctx.morph(v, "dilation", 3.0, "envelope")
    assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, 3.0, "dilation"), tol=0.0, what=f"{nx}x{ny}")
    out.free()
    v.free()
