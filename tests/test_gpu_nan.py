"""Volumes with a segment whose ends are not numbers: uploads take them, and a dilation must stay inside its
memory and leave every column out of that segment's reach as it is without it. A NaN lower end has bin 1023
of 1024, while the cover of a patch has 512 bins."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import ogrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ends", [(np.nan, 40.0), (40.0, np.nan), (np.nan, np.nan)])
@pytest.mark.parametrize("n,r", [(64, 2.0), (96, 12.0), (301, 12.0)])
def test_nan_ends_stay_local(ctx, vo, oracle, n, r, ends):
    grid, offs, z = vo.synth_volume(vo.SynthSpec(n, n_spheres=n, s_rmin=3, s_rmax=12, seed=n))
    at = int(np.nonzero(np.diff(offs) > 0)[0][np.count_nonzero(np.diff(offs) > 0) // 2])
    keep = np.ones(z.size // 2, bool)
    keep[offs[at]:offs[at + 1]] = False
    o2 = offs - np.concatenate([np.zeros(at + 1, np.int32), np.full(grid.ncols - at, offs[at + 1] - offs[at], np.int32)])
    wo, wz = oracle.morph(ogrid(oracle, grid), o2.astype(np.int32), z.reshape(-1, 2)[keep].reshape(-1), r, "dilation")
    bad = z.copy()
    bad[2 * offs[at]:2 * offs[at] + 2] = ends
    v = ctx.upload(grid, offs, bad)
    out, _ = ctx.morph(v, "dilation", r, "fast")
    go, gz = ctx.download(out)
    out.free()
    x, y = np.arange(grid.ncols) % n, np.arange(grid.ncols) // n
    for c in np.nonzero((x - at % n) ** 2 + (y - at // n) ** 2 > (r + 1) ** 2)[0]:
        assert np.array_equal(gz[2 * go[c]:2 * go[c + 1]], wz[2 * wo[c]:2 * wo[c + 1]]), c
    v.free()
