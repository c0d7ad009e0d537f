"""Every way of the integer search, each step and window pair with a tile kernel, against the FP64 oracle: the
choice by size (transforms at these sizes), the tile kernel with 16 and 24 shift columns a pass, and the direct
kernel; grids that do not fill their last tiles, regions clamped at the border, unequal extents, and radii over
one pass of shift columns.

On speckles the maximum stands alone, so all find the oracle's shift; phi comes from FP64 refits on integral
images of at most 2e5 pixels (test_gpu_search_tables.py: within 1e-8, u and v within 1e-6).
"""
import numpy as np
import pytest

import aldic_b200 as A
import oracle as O
from aldic_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,w,step,search", [
    (331, 300, 40, 10, (12, 12)), (300, 333, 40, 10, (40, 25)),
    (330, 301, 30, 16, (10, 10)), (413, 270, 30, 16, (9, 30)),
    (330, 300, 32, 16, (16, 16)), (260, 420, 32, 16, (3, 5)),
    (301, 299, 20, 12, (8, 8)), (250, 410, 20, 12, (30, 20)),
    (203, 301, 16, 9, (6, 6)), (301, 203, 16, 9, (33, 12)),
    (300, 270, 32, 8, (5, 5)), (255, 290, 32, 8, (25, 18)),
])
def test_every_way_against_the_oracle(M, N, w, step, search):
    sc = synth.temporal_affine(M=M, N=N, n_speckles=M * N // 40, u=2.4, v=-1.3, dudx=0.01, dvdy=-0.01)
    c = A.Context(0)
    try:
        c.load_image_raw(0, sc.ref, [1, M], [1, N])
        c.load_image_raw(1, sc.deff, [1, M], [1, N])
        o = O.integer_search(c.get_state(0), c.get_state(1), list(search), [1, M], [1, N], w, step)
        ok = np.isfinite(o["u"])
        assert ok.sum() > 30
        for impl, chunk, launches in ((0, 0, None), (1, 16, 11), (1, 24, 11), (2, 0, 4)):
            c.set_option(A.OPT_SEARCH_IMPL, impl)
            c.set_option(A.OPT_SEARCH_CHUNK, chunk)
            n0 = c.launches
            r = c.integer_search(list(search), [1, M], [1, N], w, step)
            assert launches in (None, c.launches - n0), (impl, chunk)  # the kernel asked for ran
            assert np.array_equal(np.isnan(r["u"]), ~ok)
            for k, tol in (("x", 0), ("y", 0), ("u", 1e-6), ("v", 1e-6), ("phi", 1e-8)):
                assert np.abs(r[k][ok] - o[k][ok]).max() <= tol, (impl, chunk, k)
    finally:
        c.close()
