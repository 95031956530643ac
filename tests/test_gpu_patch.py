"""The patch kernel of the FP32-guarded dilation at the sizes where its tiles, lists and tiers end: every
result must equal the oracle's bit for bit (the kernel decides close comparisons in FP64 and recomputes
its outputs there), through a single call and through a batch plan."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


def _columns(nx, ny, zmax, make):
    cols = [np.asarray(make(c), np.float64).reshape(-1) for c in range(nx * ny)]
    offs = np.zeros(nx * ny + 1, np.int32)
    offs[1:] = np.cumsum([c.size // 2 for c in cols])
    z = np.concatenate(cols) if offs[-1] else np.zeros(0)
    return (nx, ny, zmax), offs, z


def _random(nx, ny, zmax, most, seed, grid=None):
    rng = np.random.default_rng(seed)

    def make(_):
        k = int(rng.integers(0, most + 1))
        if grid is None:
            return np.sort(rng.uniform(0, zmax, 2 * k))
        return np.sort(rng.choice(np.arange(0, zmax, grid), 2 * k, replace=False))

    return _columns(nx, ny, zmax, make)


def _plates(nx, ny, k, pitch, thick):
    base = np.arange(k) * pitch
    return _columns(nx, ny, k * pitch, lambda c: np.stack([base, base + thick], 1))


def _thin(nx, ny, zmax, k, seed):
    rng = np.random.default_rng(seed)

    def make(_):
        z = np.sort(rng.uniform(0, zmax, k))
        return np.stack([z, z + rng.uniform(0, 0.5, k)], 1)

    return _columns(nx, ny, zmax, make)


CASES = {
    # edges of the 4 x 4 tiles and the 8 x 4 patches
    **{f"edge_{nx}x{ny}": (_random(nx, ny, 60.0, 4, nx * 100 + ny), r)
       for nx, ny, r in [(1, 1, 5.0), (5, 3, 2.25), (8, 4, 9.0), (9, 5, 12.5), (4, 33, 7.0), (37, 2, 31.0), (31, 29, 0.5)]},
    # values and radii on a lattice: ties and touches
    "ties": (_random(33, 18, 64.0, 5, 7, grid=1.0), 5.0),
    # more than 512 segments in a tile: every segment is a cluster of its own
    "dense_tile": (_random(13, 9, 4000.0, 70, 8), 6.5),
    # more than 63 components of the cover, and unions beyond 63 intervals
    "components": (_plates(20, 12, 90, 40.0, 2.0), 9.0),
    # bins much wider than the intervals: more than 1,024 of them are kept aside in a patch
    "short": (_thin(18, 11, 2.0e5, 24, 9), 3.0),
    # beyond the second tier's lists (more than 1,023 union intervals)
    "last_tier": (_plates(9, 5, 1100, 9.0, 1.0), 3.0),
    # a plane of equal ends: the nearest source alone decides
    "plane": (_columns(40, 21, 100.0, lambda c: [10.0, 20.0 + (c * 7919 % 13) / 8.0, 50.0, 50.0]), 14.5),
}


@pytest.mark.parametrize("name", list(CASES))
def test_patch_kernel_bit_exact(ctx, vo, oracle, name):
    ((nx, ny, zmax), offs, z), r = CASES[name]
    grid = vo.Grid(nx, ny, (0, 0, 0), (nx, ny, zmax), 1.0, 0)
    v = ctx.upload(grid, offs, z)
    for op in ("dilation",) if name in ("last_tier", "short") else ("dilation", "closing"):
        want = oracle.morph(ogrid(oracle, grid), offs, z, r, op)
        out, _ = ctx.morph(v, op, r, "fast")
        assert_same(ctx.download(out), want, tol=0.0, what=f"{name} {op}")
        outs, _ = ctx.morph_batched([v], [op], [r], "fast")
        assert_same(ctx.download(outs[0]), want, tol=0.0, what=f"{name} {op}, batch plan")
