"""What vo_morph_batched reports of its device time: the steps', without the planning between them."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_batched_device_time_leaves_planning_out(ctx, vo):
    """Small volumes are planned far longer than their steps run. A replay of the same steps bounds those from below; run
    one by one they have gaps between their launches, a few microseconds each."""
    vols = []
    for i in range(24):
        grid, offs, z = vo.synth_volume(vo.SynthSpec(48 + i, n_spheres=20, s_rmin=2, s_rmax=9, seed=i + 1))
        vols.append(ctx.upload(grid, offs, z))
    ops = [("dilation", "erosion", "opening", "closing")[i % 4] for i in range(24)]
    radii = [1.0 + 0.25 * i for i in range(24)]
    plan = ctx.batch(vols, ops, radii, "fast")
    replay = min(plan.run()["pass2_ms"] for _ in range(5))
    stats = plan.stats()
    plan.free()
    best = None
    for _ in range(5):
        outs, t = ctx.morph_batched(vols, ops, radii, "fast")
        for o in outs:
            o.free()
        assert t["kernel_ms"][3] == t["pass2_ms"] > 0
        best = min(best or t["pass2_ms"], t["pass2_ms"])
        total = t["total_ms"]
    for v in vols:
        v.free()
    assert best < replay + 0.02 * stats["graph_kernels"], (best, replay, total, stats["graph_kernels"])
