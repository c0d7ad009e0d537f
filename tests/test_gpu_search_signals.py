"""The integer search by transforms on signals that FP32 transforms are worst at, against the FP64 oracle: a
chirp, white noise, speckles on a steep ramp, on a large constant and beside a bright spot, and blurred
speckles, whose values fall off slowly from the peak.

The transforms' decision is certain by its error bound, so u and v are the oracle's but where the refit lies on
an edge of its rounding to 1e-3 (fewer than 1 in 200), and phi differs by the integral images' rounding alone:
45 * 2^-52 of the prefix sum of g^2 over the window's variance sum, at most 2e-8 here (the bright spot: sum
2e5 * (40 / 1)^2, variance sum 500).
"""
import numpy as np
import pytest

import aldic_b200 as A
import oracle as O
from aldic_b200 import synth_gpu

pytestmark = pytest.mark.gpu


def _blur(x, n):
    for _ in range(n):
        for ax in (0, 1):
            x = (np.roll(x, 1, ax) + 2 * x + np.roll(x, -1, ax)) / 4
    return x


def _pair(kind, M, N):
    p = synth_gpu.field_pair(9, M=M, N=N, umax=6.0, gmax=0.01)
    f, g = (im.float().cpu().numpy().reshape(M, N, order="F").astype(np.float64) for im in (p.ref, p.deff))
    f, g = (f - f.mean()) / f.std(), (g - g.mean()) / g.std()
    x, y = np.meshgrid(np.arange(M), np.arange(N), indexing="ij")
    if kind == "chirp":
        f = np.cos(2e-3 * (x ** 2 + 1.3 * y ** 2)) + 0.3 * np.sin(1.1e-3 * (x - y) ** 2)
        g = np.roll(f, (3, -4), (0, 1))
    elif kind == "noise":
        f = np.random.default_rng(0).normal(size=(M, N))
        g = np.roll(f, (-5, 2), (0, 1))
    elif kind == "ramp":
        f, g = f + 0.2 * x, g + 0.2 * x
    elif kind == "constant":
        f, g = f + 60, g + 60
    elif kind == "spot":
        g[M // 2:M // 2 + 9, N // 2:N // 2 + 9] = f[M // 2:M // 2 + 9, N // 2:N // 2 + 9] = 40
    elif kind == "blurred":
        f, g = _blur(f, 60), _blur(g, 60)
        f, g = f / f.std(), g / g.std()
    return f.astype(np.float32), g.astype(np.float32)


@pytest.mark.parametrize("kind", ["chirp", "noise", "ramp", "constant", "spot", "blurred"])
@pytest.mark.parametrize("M,N,w,step,r", [(330, 360, 24, 9, 10), (400, 380, 40, 14, 33)])
def test_hard_signals(kind, M, N, w, step, r):
    f, g = _pair(kind, M, N)
    c = A.Context(0)
    try:
        c.load_image(0, f)
        c.load_image(1, g)
        got = c.integer_search([r, r], [1, M], [1, N], w, step)
        print(kind, "left", c.get_option(A.STAT_SEARCH_LEFT), "of", got["u"].size)
    finally:
        c.close()
    o = O.integer_search(f.astype(np.float64), g.astype(np.float64), [r, r], [1, M], [1, N], w, step)
    assert np.array_equal(np.isnan(got["u"]), np.isnan(o["u"]))
    d = np.maximum(np.abs(got["u"] - o["u"]), np.abs(got["v"] - o["v"]))
    assert np.nanmax(d) <= 1e-3 + 1e-9 and np.mean(d > 1e-9) < 0.005
    same = d <= 1e-9
    assert np.abs(got["phi"] - o["phi"])[same].max() <= 2e-8
