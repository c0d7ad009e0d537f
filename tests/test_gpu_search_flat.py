"""The integer search by transforms on frames with areas of one value (a saturated or clipped background,
a mask multiplied into the raw frames): windows there have no variance and must neither win nor send their
subsets to the direct sums.

Against the FP64 oracle as test_gpu_search_fft.py's constant background: at most 0.5 % of the subsets, those
on the edge of an area, may differ, and no more than with the direct kernel.  Left to direct sums: subsets
with several shifts within the transforms' error of one another, none on speckles; 0.5 % is allowed.
"""
import numpy as np
import pytest

import aldic_b200 as A
import oracle as O
from aldic_b200 import synth_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,w,step,search,value,bits", [
    (400, 410, 40, 10, 30, 0, 8),
    (400, 410, 40, 10, 30, 255, 8),
    (400, 410, 24, 7, 20, 0, 16),
    (640, 330, 32, 16, 20, 131, 16),
    (330, 520, 60, 13, 33, 0, 8),
])
def test_constant_areas(M, N, w, step, search, value, bits):
    p = synth_gpu.field_pair(5, M=M, N=N, umax=0.5 * search, gmax=0.03)
    x, y = np.meshgrid(np.arange(M), np.arange(N), indexing="ij")
    area = (x < M // 7) | (y > N - N // 8)
    for cx, cy, r in ((0.6, 0.4, 0.13), (0.35, 0.65, 0.1), (0.8, 0.75, 0.08)):
        area |= (x - cx * M) ** 2 + (y - cy * N) ** 2 < (r * min(M, N)) ** 2
    scale = 200 if bits == 16 else 1
    rng = np.random.default_rng(0)
    c = A.Context(0)
    try:
        for slot, im in enumerate((p.ref, p.deff)):
            im = im.cpu().numpy().reshape(M, N, order="F").astype(np.int64) * scale
            im += rng.integers(0, scale, im.shape)
            im[area] = value * scale
            c.load_image_raw(slot, im.astype(np.uint16 if bits == 16 else np.uint8), [1, M], [1, N])
        f, g = c.get_state(0), c.get_state(1)
        o = O.integer_search(f, g, [search] * 2, [1, M], [1, N], w, step)
        off = {}
        for impl in (0, 2):
            c.set_option(A.OPT_SEARCH_IMPL, impl)
            r = c.integer_search([search] * 2, [1, M], [1, N], w, step)
            left = c.get_option(A.STAT_SEARCH_LEFT)
            assert np.array_equal(np.isnan(r["u"]), np.isnan(o["u"]))
            off[impl] = int(np.sum(np.any([np.abs(r[k] - o[k]) > 1e-3 + 1e-9 for k in ("u", "v")], 0)))  # subsets
            assert left <= 0.005 * o["u"].size, (impl, left)
        assert off[0] <= off[2] + 2 and off[0] <= 0.005 * o["u"].size, off
    finally:
        c.close()
