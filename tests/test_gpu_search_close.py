"""Shifts whose normalised values differ by less than an FP32 number resolves: the integer search by transforms
decides them in FP64.

A pattern of period 16 plus noise of relative size e, searched for in itself: the value is 1 at shift 0 and
1 / (1 + e^2) at the other repeats, 1.4e-8 to 4e-8 below, where FP32 numbers just under 1 lie 6e-8 apart.  FP64
values are off by some 1e-12 on frames of this size.  Without noise the repeats are equal, and the first shift in
column-major order within the search wins: the one at the smallest offsets, -16.
"""
import numpy as np
import pytest

import aldic_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,w,step,r,e", [(400, 410, 24, 11, 20, 1.2e-4), (400, 410, 40, 9, 20, 2e-4),
                                            (300, 500, 24, 11, 20, 0.0)])
def test_close_values(M, N, w, step, r, e):
    rng = np.random.default_rng(1)
    t = rng.integers(-4, 5, (16, 16)) * 0.25
    f = np.tile(t / t.std(), (M // 16 + 1, N // 16 + 1))[:M, :N]
    f = (f + e * rng.normal(size=f.shape)).astype(np.float32)
    c = A.Context(0)
    try:
        for slot in (0, 1):
            c.load_image(slot, f)
        o = c.integer_search([r, r], [1, M], [1, N], w, step)
        assert c.get_option(A.STAT_SEARCH_LEFT) == 0
    finally:
        c.close()
    inner = (o["x"] - w // 2 - r > 0) & (o["x"] + w // 2 + r < M) & (o["y"] - w // 2 - r > 0) & (o["y"] + w // 2 + r < N)
    assert inner.sum() > 50
    want = 0.0 if e else -16.0
    for k in ("u", "v"):
        assert np.abs(o[k][inner] - want).max() < 0.05, k
