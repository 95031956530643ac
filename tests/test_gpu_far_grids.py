"""Volumes far from z = 0: the filters take their values relative to the grid's origin. Origins that fit the values,
origins that do not (nothing is passed over by mistake then either), both signs. The oracle's own FP64 candidates, so
equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift,origin", [(50000.0, 50000.0), (1e6 + 0.3, 1e6), (-1e7, -1e7), (1e7, 0.0), (0.0, 1e7), (3e11, 3e11),
                                          (1e6, -1e6), (0.25, 1e300)])
@pytest.mark.parametrize("n,r,method", [(70, 3.0, "fast"), (300, 5.0, "fast"), (140, 14.0, "fast"), (300, 20.0, "fast"),
                                        (110, 9.0, "envelope"), (520, 5.0, "fast")])
def test_far_grids(ctx, vo, oracle, n, r, method, shift, origin):
    g, offs, z = vo.synth_volume(vo.SynthSpec(n, n_spheres=n * n // 250, s_rmin=2, s_rmax=max(8, n / 12), n_cyl=n // 10, seed=n))
    z = z + shift
    grid = vo.Grid(n, n, (0, 0, origin), g.extent, 1.0, 0)
    want = oracle.morph(ogrid(oracle, grid), offs, z, r, "dilation")
    v = ctx.upload(grid, offs, z)
    out, _ = ctx.morph(v, "dilation", r, method)
    assert_same(ctx.download(out), want, tol=0.0, what=f"{n} r={r} {method} z + {shift}")
    out.free()
    if method == "fast":
        outs, _ = ctx.morph_batched([v], ["dilation"], [r], "fast")
        assert_same(ctx.download(outs[0]), want, tol=0.0, what=f"batch {n} r={r} z + {shift}")
        outs[0].free()
    v.free()
