"""The integer search by transforms against the direct per-subset correlation, for every transform size
(48 to 192) at its smallest and largest crop, odd windows and steps, clamped search regions, unequal
extents, masked frames, a constant background, a repeating pattern and values that are not finite.

Both find the first maximum of the same function and fit it in FP64: u and v are a whole shift plus a
fit rounded to 1e-3, so equal unless the fit lies on a rounding edge; phi differs by the order of FP64
sums over at most 121^2 products: 1.5e4 * 2^-53 < 2e-12.
"""
import numpy as np
import pytest

import aldic_b200 as A
import oracle as O
from aldic_b200 import synth_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


def pair(M, N, umax, seed=4):
    p = synth_gpu.field_pair(seed, M=M, N=N, umax=umax, gmax=0.05)
    f, g = (im.float().cpu().numpy().reshape(M, N, order="F") for im in (p.ref, p.deff))
    return [((im - im.mean()) / im.std()).astype(np.float32) for im in (f, g)]


def run(ctx, f, g, search, w, step):
    M, N = f.shape
    ctx.load_image(0, f)
    ctx.load_image(1, g)
    r = {}
    for impl in (0, 2):
        ctx.set_option(A.OPT_SEARCH_IMPL, impl)
        n0 = ctx.launches
        r[impl] = ctx.integer_search(list(search), [1, M], [1, N], w, step)
        r[impl]["launches"] = ctx.launches - n0
    ctx.set_option(A.OPT_SEARCH_IMPL, 0)
    # another kernel than the direct one, unless the template leaves no room for the transform
    assert (r[0].pop("launches") > r[2].pop("launches")) == (w < 118)
    return r


def check(r):
    for k in ("u", "v"):
        a, b = r[0][k], r[2][k]
        assert np.array_equal(np.isnan(a), np.isnan(b)), k
        d = np.abs(a - b)[~np.isnan(a)]
        assert d.size and d.max() <= 1e-3 + 1e-9 and np.mean(d > 1e-9) < 1e-3, (k, d.max(), np.mean(d > 1e-9))
    np.testing.assert_allclose(r[0]["phi"], r[2]["phi"], atol=2e-12)


def both(*a):
    check(run(*a))


@pytest.mark.parametrize("M,N,w,step,search", [
    (420, 431, 20, 5, (4, 4)),       # 48
    (401, 422, 18, 5, (14, 14)),     # 48, its largest crop
    (420, 431, 26, 5, (11, 11)),     # 48 + 2: 64
    (333, 421, 22, 7, (20, 20)),     # 64, its largest
    (300, 421, 30, 7, (24, 24)),     # 80, its largest
    (300, 391, 24, 11, (20, 37)),    # unequal extents: 96
    (311, 300, 44, 11, (24, 24)),    # 96, its largest
    (311, 300, 60, 13, (33, 32)),    # 128, its largest
    (412, 300, 26, 13, (58, 58)),    # 144, its largest
    (397, 420, 48, 21, (50, 55)),    # 160
    (431, 420, 50, 19, (70, 70)),    # 192, its largest
    (400, 410, 118, 27, (20, 21)),   # 192 with this template is more than the shared memory
    (411, 400, 76, 27, (20, 21)),    # 128, a template of three 32-row groups
    (260, 270, 40, 31, (70, 70)),    # every subset's region clamped
    (640, 640, 40, 10, (70, 70)),    # a pair that has a tile kernel
    (512, 300, 30, 16, (10, 10)),
])
def test_against_direct(ctx, M, N, w, step, search):
    f, g = pair(M, N, 0.6 * min(search))
    both(ctx, f, g, search, w, step)


def test_masked_and_periodic(ctx):
    f, g = pair(400, 410, 8.0)
    f[150:260, 120:240] = g[150:260, 120:240] = 0  # under a mask
    both(ctx, f, g, (20, 20), 24, 7)
    t = np.random.default_rng(0).integers(-4, 5, (16, 16)).astype(np.float32) * 0.25
    p = np.tile(t, (26, 26))  # the maximum, 1, repeats 16 pixels on
    r = run(ctx, p, p, (20, 20), 24, 11)
    # FP32 sums can round a value of 1 to more than 1, which counts as 0: the direct kernel then takes
    # another shift.  Here the close ones are decided in FP64.
    for k in ("u", "v"):
        d = r[0][k] - 16 * np.round(r[0][k] / 16)
        assert np.nanmax(np.abs(d)) < 0.05, k
    assert np.nanmin(r[0]["phi"] - r[2]["phi"]) > -1e-9


def test_constant_background(ctx):
    """Windows whose variance sum is all cancellation: the direct kernel's FP32 sums can exceed it, so
    both are held against the FP64 oracle."""
    f, g = pair(400, 410, 8.0)
    f[150:260, 120:240] = g[150:260, 120:240] = 0
    f[:, 300:] = g[:, 300:] = -2.125
    r = run(ctx, f, g, (20, 20), 24, 7)
    o = O.integer_search(f.astype(np.float64), g.astype(np.float64), [20, 20], [1, 400], [1, 410], 24, 7)
    off = {i: sum(int(np.sum(np.abs(r[i][k] - o[k]) > 1e-3 + 1e-9)) for k in ("u", "v")) for i in r}
    assert off[0] <= off[2] <= 0.005 * o["u"].size, off
    assert np.array_equal(np.isnan(r[0]["u"]), np.isnan(o["u"]))


def test_not_finite(ctx):
    f, g = pair(400, 410, 8.0)
    g[210, 190] = np.nan
    both(ctx, f, g, (20, 20), 24, 7)
    g[210, 190] = 0
    g[333, 317] = np.inf
    both(ctx, f, g, (20, 20), 24, 7)
