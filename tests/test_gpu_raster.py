"""Dexelization facet by facet: facets of one column, of a warp's and of more than one warp takes, at the
ends of each range; hits that fit a column's slots and that do not; meshes with no hits. The oracle makes the
same FP64 operations column by column, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_same

pytestmark = pytest.mark.gpu


def check(ctx, oracle, verts, tris, **kw):
    verts, tris = np.ascontiguousarray(verts, dtype=np.float64), np.ascontiguousarray(tris, dtype=np.int32)
    _, offs, z = oracle.dexelize(verts, tris, **kw)
    v = ctx.dexelize(verts, tris, **kw)
    assert_same(ctx.download(v), (offs, z), tol=0.0)
    v.free()
    return np.diff(offs)


def sheet(n, m, size, level, rng, rough):
    """An n x m grid of quads over `size`, with heights around `level`."""
    x, y = np.meshgrid(np.linspace(0, size[0], n + 1), np.linspace(0, size[1], m + 1), indexing="ij")
    v = np.stack([x, y, level + rough * rng.random(x.shape)], -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(n), np.arange(m), indexing="ij")
    a = (i * (m + 1) + j).reshape(-1)
    return v, np.concatenate([np.stack([a, a + m + 1, a + 1], 1), np.stack([a + 1, a + m + 1, a + m + 2], 1)])


def stack(sheets):
    vs, ts, n = [], [], 0
    for v, t in sheets:
        vs.append(v)
        ts.append(t + n)
        n += len(v)
    return np.concatenate(vs), np.concatenate(ts)


@pytest.mark.parametrize("n,m,dexels", [(1, 1, 40), (1, 1, 130), (1, 1, 64), (2, 1, 90), (20, 16, 60), (20, 16, 75),
                                        (40, 40, 30), (3, 50, 200)])
def test_raster_facet_sizes(ctx, oracle, n, m, dexels):
    rng = np.random.default_rng(n * 1000 + dexels)
    mesh = stack([sheet(n, m, (1.0, 0.83), 0.2, rng, 0.1), sheet(m, n, (1.0, 0.83), 0.6, rng, 0.1)])
    assert check(ctx, oracle, *mesh, num_dexels=dexels, padding=2).sum() > 0


@pytest.mark.parametrize("layers", [1, 15, 16, 17, 33, 130])
def test_raster_hits_per_column(ctx, oracle, layers):
    """Up to `layers` hits, unsorted in the mesh; an odd count leaves one unpaired."""
    rng = np.random.default_rng(layers)
    levels = rng.permutation(layers) + 1.0
    mesh = stack([sheet(2, 3, (20.0 - 3 * (i % 4), 14.0), levels[i], rng, 0.3) for i in range(layers)])
    got = check(ctx, oracle, *mesh, num_dexels=-1, padding=1, spacing=1.0)
    assert got.max() == layers // 2


def test_raster_refuses_too_many_hits(ctx, vo):
    rng = np.random.default_rng(1)
    mesh = stack([sheet(1, 1, (3.0, 3.0), 1.0 + 0.01 * i, rng, 0.0) for i in range(4098)])
    with pytest.raises(Exception, match="4096"):
        ctx.dexelize(np.ascontiguousarray(mesh[0]), np.ascontiguousarray(mesh[1], dtype=np.int32), num_dexels=-1,
                     padding=0, spacing=1.0)
    with pytest.raises(Exception):
        ctx.dexelize_odd_columns()
