"""The envelope form's sweeps in segments of lines and rows, and its ends held as ordered integers:
lengths at which the split begins or leaves a remainder, radii whose reach crosses the segment ends,
segments re-run with global-memory state, and ends of either sign, signed zeros and large magnitudes.
The union is of the oracle's own FP64 candidates, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


def check(ctx, oracle, grid, offs, z, op, r):
    v = ctx.upload(grid, offs, z)
    out, t = ctx.morph(v, op, r, "envelope")
    assert t["mid_pieces"] > 0
    assert_same(ctx.download(out), oracle.morph(ogrid(oracle, grid), offs, z, r, op), tol=0.0, what=f"{op} r={r}")
    out.free()
    v.free()
    return t


@pytest.mark.parametrize("nx,ny,r", [(31, 63, 0.5), (33, 64, 2.0), (64, 65, 4.0), (129, 7, 4.5), (5, 260, 8.5), (200, 3, 11.0)])
def test_envelope_segment_edges(ctx, vo, oracle, nx, ny, r, monkeypatch):
    n = max(nx, ny)
    grid, offs, z = vo.synth_volume(vo.SynthSpec(nx, ny=ny, n_spheres=30, s_rmin=1, s_rmax=n / 6, n_cyl=5, seed=nx))
    for op in ("dilation", "erosion"):
        check(ctx, oracle, grid, offs, z, op, r)
    monkeypatch.setenv("VO_ENVELOPE_STATE_CAP", "4")  # every row segment re-runs
    t = check(ctx, oracle, grid, offs, z, "dilation", r)
    assert t["overflow_columns"] > 0 or r < 1  # below that a state is one column's pieces


@pytest.mark.parametrize("shift,scale", [(-40.0, 1.0), (0.0, 1e-3), (-1e12, 1.0), (1e-310, 1e-300), (0.0, 1e39)])
def test_envelope_ends_of_any_sign_and_size(ctx, vo, oracle, shift, scale):
    rng = np.random.default_rng(3)
    nx, ny, k = 70, 66, 3
    e = np.cumsum(rng.integers(1, 60, (nx * ny, 2 * k)), axis=1).astype(np.float64) / 4 * scale + shift
    e[::7] -= e[::7, 2:3]
    e[::7, 2] = -0.0
    offs = (np.arange(nx * ny + 1) * k).astype(np.int32)
    top = max(1.0, float(np.abs(e).max()) * 2)
    grid = vo.Grid(nx, ny, (0, 0, -top), (nx, ny, 2 * top), 1.0, 0)
    check(ctx, oracle, grid, offs, np.ascontiguousarray(e).reshape(-1), "dilation", 3.5)
