"""The shape that a plan reports of its main kernel is that of the kernel which ran."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


# small radius; patches, with four lanes per column and with one; smooth and dense: column by column
@pytest.mark.parametrize("n,spheres,r,lanes,slots,persistent", [(64, 40, 3.0, 4, 48, 0), (300, 300, 3.0, 1, 48, 0),
                                                                (64, 40, 20.0, 4, 64, 1), (900, 600, 24.0, 1, 64, 1),
                                                                (700, 2000, 6.0, 1, 24, 0)])
def test_reported_kernel_shape(ctx, vo, n, spheres, r, lanes, slots, persistent):
    grid, offs, z = vo.synth_volume(vo.SynthSpec(n, n_spheres=spheres, s_rmin=2, s_rmax=max(8, min(40, n // 8)), seed=n))
    v = ctx.upload(grid, offs, z)
    plan = ctx.batch([v], ["dilation"], [r], "fast")
    s = plan.stats()
    plan.free()
    v.free()
    assert (s["tile_rows"], s["persistent"]) == (lanes, persistent), s
    assert s["union_cap"] == slots, s
    assert 16 <= s["regs"] <= 128
