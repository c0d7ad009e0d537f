"""The tables the integer search is built on (integral images in 64 x 64 tiles, window maps in 32 x 32
tiles with the largest value of every 16 positions, ring columns in passes of 512 shifts) at the sizes
where their tiles end: whole tiles, one row or column more, images of one tile, more columns than a
prefix block holds, and a search over more shifts than one pass.

The peak's FP64 refit reads the integral images at the window sums' own precision: prefix sums over at
most 4e5 pixels of O(1) values lose no more than 4e5 * 2^-53 * 4e5 / (window variance sum > 1) < 2e-5 in
the worst case and about sqrt of it, 4e-9, as they round: phi within 1e-8, u and v (integer peak plus a
quadratic fit of phi) within 1e-6.
"""
import numpy as np
import pytest

import oracle as O
from aldic_b200 import Context, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)  # one context: its buffers go from shape to shape
    yield c
    c.close()


@pytest.mark.parametrize("M,N,w,st,search", [
    (64, 640, 16, 9, (4, 4)),
    (600, 65, 16, 9, (4, 4)),     # a smaller area than the one before, more tile rows
    (128, 128, 20, 12, (6, 6)),
    (129, 127, 20, 12, (6, 6)),
    (65, 1100, 30, 16, (5, 5)),   # columns beyond one prefix block of 1024
    (64, 64, 32, 16, (3, 3)),
    (63, 64, 24, 7, (3, 5)),      # no tile kernel: integral images alone
    (160, 150, 16, 9, (280, 260)),  # 543 shifts: two passes of the ring columns
])
def test_search_tables(ctx, M, N, w, st, search):
    sc = synth.temporal_affine(M=M, N=N, n_speckles=max(60, M * N // 40), u=1.4, v=-1.3)
    ctx.load_image_raw(0, sc.ref, [1, M], [1, N])
    ctx.load_image_raw(1, sc.deff, [1, M], [1, N])
    ctx.set_mask(None)
    ctx.compute_gradients()
    f, g = ctx.get_state(0), ctx.get_state(1)
    r = ctx.integer_search(list(search), [1, M], [1, N], w, st)
    ro = O.integer_search(f, g, list(search), [1, M], [1, N], w, st)
    assert np.array_equal(np.isnan(r["u"]), np.isnan(ro["u"]))
    ok = np.isfinite(ro["u"])
    assert ok.any()
    for k in ("u", "v"):
        assert np.max(np.abs(r[k][ok] - ro[k][ok])) < 1e-6, k
    assert np.max(np.abs(r["phi"][ok] - ro["phi"][ok])) < 1e-8
