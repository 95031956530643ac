"""The columns kernel: inputs that take it first (smooth, dense, small radius, at least 2^18 columns), and unions
of more intervals than the lists of the small-radius and patch kernels hold, in few columns, in many and in most:
by its second launch, by the FP64 tier, or all over again. Single calls, replayed plans and batches against the
oracle's own FP64 candidates, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same, ogrid

pytestmark = pytest.mark.gpu


def scattered(vo, nx, ny, per, height, length, seed, where=None):
    """Columns of Poisson(per) segments up to `length` long, anywhere in [0, height); `where`: other counts for some."""
    rng = np.random.default_rng(seed)
    count = rng.poisson(per, nx * ny)
    if where is not None:
        count[rng.choice(nx * ny, where[0], replace=False)] = where[1]
    offs = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
    lo = rng.uniform(0, height, offs[-1])
    col = np.repeat(np.arange(nx * ny), count)
    lo = lo[np.lexsort((lo, col))]
    nxt = np.append(lo[1:], np.inf)
    nxt[offs[1:][count > 0] - 1] = np.inf
    hi = np.minimum(lo + rng.uniform(0, length, lo.size), lo + 0.9 * (nxt - lo))
    return vo.Grid(nx, ny, (0, 0, 0), (nx, ny, height), 1.0, 0), offs, np.stack([lo, hi], 1).reshape(-1)


def check(ctx, oracle, grid, offs, z, r, op="dilation", what=""):
    want = oracle.morph(ogrid(oracle, grid), offs, z, r, op)
    v = ctx.upload(grid, offs, z)
    out, t = ctx.morph(v, op, r, "fast")
    assert_same(ctx.download(out), want, tol=0.0, what=f"{what} morph r={r}")
    plan = ctx.batch([v], [op], [r])
    for _ in range(2):
        plan.run()
        outs = plan.outputs()
        assert_same(ctx.download(outs[0]), want, tol=0.0, what=f"{what} plan r={r}")
        outs[0].free()
    plan.free()
    outs, _ = ctx.morph_batched([v, v], [op, op], [r, r], "fast")
    for o in outs:
        assert_same(ctx.download(o), want, tol=0.0, what=f"{what} batch r={r}")
        o.free()
    out.free()
    v.free()
    return t


# sides that leave remainders of the 8 x 4 patches and of the 512-column bands
@pytest.mark.parametrize("nx,ny,spheres,r", [(513, 515, 1300, 5.0), (1030, 261, 1500, 6.25), (512, 512, 1600, 4.5), (4097, 66, 1200, 7.0)])
def test_smooth_dense_volumes(ctx, vo, oracle, nx, ny, spheres, r):
    grid, offs, z = vo.synth_volume(vo.SynthSpec(nx, ny=ny, zmax=512.0, n_spheres=spheres, s_rmin=3, s_rmax=38, seed=nx))
    for op in ("dilation", "closing"):
        check(ctx, oracle, grid, offs, z, r, op, what=f"{nx}x{ny}")


@pytest.mark.parametrize("nx,ny", [(64, 64), (131, 97), (300, 5), (1, 700)])
@pytest.mark.parametrize("per,height,r", [(12, 3000.0, 1.0), (12, 3000.0, 2.0), (4, 2000.0, 4.0), (3, 9000.0, 9.0), (2, 4000.0, 14.5)])
def test_unions_beyond_the_lists(ctx, vo, oracle, nx, ny, per, height, r):
    check(ctx, oracle, *scattered(vo, nx, ny, per, height, 1.0, nx + int(r)), r, what=f"{nx}x{ny} per={per}")


# a few columns, more than kFewColumns of them, and too many, with unions of 64..127, 128.. and over 1024 intervals
@pytest.mark.parametrize("where", [(3, 60), (60, 60), (900, 60), (30, 200), (6, 1500)])
@pytest.mark.parametrize("n,r", [(150, 0.5), (150, 3.0), (150, 13.0), (600, 2.0)])
def test_some_columns_of_many_segments(ctx, vo, oracle, n, r, where):
    check(ctx, oracle, *scattered(vo, n, n, 0.4, 20000.0, 2.0, n, where), r, what=f"{n} {where}")
