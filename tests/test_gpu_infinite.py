"""Columns with infinite ends, or ends far beyond the others: a dilation keeps them, and bins and FP32 copies
of the rest must not suffer. The oracle's own FP64 candidates, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import ogrid

pytestmark = pytest.mark.gpu


def volume(vo, n, low, high):
    """Spheres; the lowest segment of every seventh column that has one reaches down to `low`, the highest of every
    fifth up to `high`, and some columns have segments beyond everything else."""
    grid, offs, z = vo.synth_volume(vo.SynthSpec(n, n_spheres=n, s_rmin=4, s_rmax=max(8, n / 6), n_cyl=n // 8, seed=n))
    z = z.reshape(-1, 2).copy()
    have = np.nonzero(np.diff(offs) > 0)[0]
    if low is not None:
        z[offs[have[::7]], 0] = low
        if np.isfinite(low):  # the oracle's painter has no place for a point at minus infinity
            z[offs[have[3::97]]] = [low, low]
    if high is not None:
        z[offs[have[::5] + 1] - 1, 1] = high
    return grid, offs, np.ascontiguousarray(z.reshape(-1))


@pytest.mark.parametrize("low,high", [(-np.inf, None), (None, np.inf), (-np.inf, np.inf), (-1e36, 1e33), (-3e25, 4e18),
                                      (-1e300, np.inf)])
@pytest.mark.parametrize("n,r", [(48, 2.0), (48, 20.5), (96, 12.0), (300, 12.0), (300, 33.0)])
def test_infinite_ends(ctx, vo, oracle, n, r, low, high):
    grid, offs, z = volume(vo, n, low, high)
    want = oracle.morph(ogrid(oracle, grid), offs, z, r, "dilation")
    v = ctx.upload(grid, offs, z)
    out, _ = ctx.morph(v, "dilation", r, "fast")
    plan = ctx.batch([v], ["dilation"], [r])
    plan.run()
    outs = plan.outputs()
    for what, o in (("morph", out), ("plan", outs[0])):
        go, gz = ctx.download(o)
        assert np.array_equal(go, want[0]), what
        assert np.array_equal(gz, want[1]), what
        o.free()
    plan.free()
    v.free()
