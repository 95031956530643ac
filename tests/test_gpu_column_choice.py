"""Which kernel a dilation by a small radius takes first does not hang on how the growths of H fall at one radius: smooth
dense volumes go column by column, thin cylinders do not, and no sample is taken of what is done sooner."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

DIRECT, COLUMNS = 48, (24, 32)  # union slots per column of the two kernels


def slots(ctx, grid, offs, z, r):
    v = ctx.upload(grid, offs, z)
    plan = ctx.batch([v], ["dilation"], [r])
    plan.run()
    s = plan.stats()
    plan.free()
    v.free()
    return s["union_cap"]


@pytest.mark.parametrize("r", [4.5, 5.0, 5.5, 6.0])
def test_by_the_kind_of_volume(ctx, vo, r):
    grid, offs, z = vo.synth_volume(vo.SynthSpec(700, n_spheres=0, n_cyl=900, seed=6))
    assert slots(ctx, grid, offs, z, r) == DIRECT
    grid, offs, z = vo.synth_volume(vo.SynthSpec(700, n_spheres=2500, s_rmin=3, s_rmax=35, seed=6))
    assert slots(ctx, grid, offs, z, r) in COLUMNS


def test_no_sample_of_short_calls(ctx, vo):
    grid, offs, z = vo.synth_volume(vo.SynthSpec(512, n_spheres=0, n_cyl=500, seed=6))
    v = ctx.upload(grid, offs, z)
    ctx.morph(v, "dilation", 3.0, "fast")[0].free()  # the first use of a volume looks for inverted pairs besides
    counts = []
    for r in (3.0, 5.0, 6.0):
        out, t = ctx.morph(v, "dilation", r, "fast")
        counts.append(t["kernel_launches"])
        out.free()
    v.free()
    assert counts[0] == counts[1] == counts[2]
