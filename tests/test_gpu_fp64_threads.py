"""ALDIC_OPT_FP64_THREADS splits the FP64 re-solve's sums over the threads it names: the codes do not depend
on it, the converged displacements only in the last digits.

Sums of at most 41^2 products in another order differ by 1e-13 of their size; the solve's condition (the
window's texture against its size) carries that to below 1e-9 px.  That no subset of some hundred keeps all
its bits when the order changes is what shows that another split ran.
"""
import numpy as np
import pytest

import aldic_b200 as A
from aldic_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,w,default", [(0, 20, 128), (1, 22, 128), (0, 24, 256), (1, 40, 256), (1, 50, 256), (0, 52, 512)])
def test_threads_of_the_fp64_pass(variant, w, default):
    sc = synth.temporal_affine(M=270, N=250, n_speckles=1400, u=2.3, v=-1.4, dudx=0.02, dvdy=-0.015)
    M, N = sc.ref.shape
    c = A.Context(0)
    try:
        c.load_image_raw(0, sc.ref, [1, M], [1, N])
        c.load_image_raw(1, sc.deff, [1, M], [1, N])
        c.compute_gradients()
        x, y = np.meshgrid(np.arange(40, M - 40, 14.0), np.arange(40, N - 40, 14.0), indexing="ij")
        nodes = np.stack([x.ravel(), y.ravel()], 1)
        u, v = sc.disp(nodes[:, 0], nodes[:, 1])
        U0 = np.stack([np.round(u), np.round(v)], 1).ravel()
        c.set_fp64_band(1e30)  # every subset is re-solved in FP64
        assert c.get_option(A.OPT_FP64_THREADS) == 0
        r = {0: c.local_icgn(variant, nodes, U0, w, 1e-3)}
        for n in (128, 256, 512):
            c.set_option(A.OPT_FP64_THREADS, n)
            r[n] = c.local_icgn(variant, nodes, U0, w, 1e-3)
            assert c.get_option(A.STAT_FP64_RESOLVES) == len(nodes)
            assert np.array_equal(r[n]["conv"], r[0]["conv"])
            assert np.abs(r[n]["U"] - r[0]["U"]).max() < 1e-9
        assert np.array_equal(r[default]["U"], r[0]["U"])
        assert not np.array_equal(r[128]["U"], r[512]["U"]) and not np.array_equal(r[256]["U"], r[512]["U"])
        c.set_option(A.OPT_FP64_THREADS, 0)  # back to the default
        assert np.array_equal(c.local_icgn(variant, nodes, U0, w, 1e-3)["U"], r[0]["U"])
        for bad in (64, 1024, -1):
            with pytest.raises(A.AldicError):
                c.set_option(A.OPT_FP64_THREADS, bad)
    finally:
        c.close()
