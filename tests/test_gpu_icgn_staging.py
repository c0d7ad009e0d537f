"""IC-GN at the edges of the staging rule: the last window that is always staged (45 pixels), the first that is
staged only where its subsets run at once, the last of those (69) and the first that never is (71), with n at and
above the number that runs at once (2 subsets a CTA, 6 or 4 CTAs an SM, 148 SMs).  Where the taps are read does
not change their values: equal to the bit with ALDIC_OPT_STAGING, which stages every window that fits.
"""
import numpy as np
import pytest

import aldic_b200 as A
from aldic_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,ctas", [(44, 8), (46, 6), (68, 4), (70, 3)])
@pytest.mark.parametrize("variant", [0, 1])
def test_staging_changes_no_bit(w, ctas, variant):
    sc = synth.temporal_affine(M=270, N=250, n_speckles=1400, u=2.3, v=-1.4, dudx=0.02, dvdy=-0.015)
    M, N = sc.ref.shape
    rng = np.random.default_rng(w)
    c = A.Context(0)
    try:
        c.load_image_raw(0, sc.ref, [1, M], [1, N])
        c.load_image_raw(1, sc.deff, [1, M], [1, N])
        c.compute_gradients()
        at_once = 2 * ctas * 148
        h = w // 2 + 8
        xy = np.stack([rng.integers(h, M - h, at_once + 1), rng.integers(h, N - h, at_once + 1)], 1).astype(float)
        u, v = sc.disp(xy[:, 0], xy[:, 1])
        U0 = np.stack([np.round(u, 1), np.round(v, 1)], 1).ravel()
        out = {}
        for staging in (0, 1):
            c.set_option(A.OPT_STAGING, staging)
            for n in (at_once, at_once + 1):
                out[staging, n] = c.local_icgn(variant, xy[:n], U0[:2 * n], w, 1e-3)
        for (staging, n), r in out.items():
            assert np.mean((r["conv"] > 0) & (r["conv"] < 100)) > 0.95
            for k, per in (("U", 2), ("F", 4), ("conv", 1)):
                a, b = np.asarray(r[k]).ravel(), np.asarray(out[0, at_once + 1][k]).ravel()
                assert np.array_equal(a[:per * at_once], b[:per * at_once], equal_nan=True), (staging, n, k)
    finally:
        c.close()
