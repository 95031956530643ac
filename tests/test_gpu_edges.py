"""Branches of the 2D image path and of the sizer's training kernels at the sizes where they begin:
results larger than the image staging buffer, and sample counts that leave remainders of every tile."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spans,h,r", [(1000, 20, 5.0), (1000, 20, 0.5), (1, 1, 3.0)])
def test_image_result_beyond_staging(ctx, oracle, spans, h, r):
    """One row of narrow spans 12 pixels apart: a dilation by 5 copies them to 11 rows, more events than
    the buffer sized for the input's; whole numbers, so equality is exact."""
    w = 12 * spans + 8
    ev = np.stack([4 + 12 * np.arange(spans), 5 + 12 * np.arange(spans)], 1).reshape(-1).astype(np.int32)
    offs = np.zeros(h + 1, np.int32)
    offs[h // 2 + 1:] = ev.size
    for op, name in (("dilation", "dilate"), ("erosion", "erode"), ("closing", "close")):
        got = ctx.image_morph(w, h, offs, ev, r, op)
        want = oracle.image_morph(w, h, offs, ev, r, name)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), op


@pytest.mark.parametrize("n", [1, 3, 31, 513, 39001])
def test_sizer_gradients_at_tile_remainders(ctx, vo, n):
    """Against the numpy oracle of the same BF16 network in FP64: FP32 sums over n samples, 2e-4 of the
    largest component as in the gradient test of the sizer."""
    from oracle import sizer_oracle as S
    rng = np.random.default_rng(n)
    X = rng.normal(0, 1, (n, vo.SIZER_FEATURES)).astype(np.float32)
    T = rng.uniform(0, 6, (n, vo.SIZER_OUTPUTS)).astype(np.float32)
    sz = ctx.sizer(seed=5)
    g, loss = sz.gradients(X, T)
    want_loss, want = S.loss_and_gradients(sz.params(), X, T)
    assert abs(loss - want_loss) <= 1e-4 * max(1.0, want_loss)
    assert np.abs(g - want).max() <= 2e-4 * np.abs(want).max()
    pred = sz.forward(X)
    assert np.array_equal(pred, sz.forward(X))
    sz.free()
