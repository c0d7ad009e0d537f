"""The autotuner's report of the search: the choice by size is timed and named with the kernel that it takes,
and the other candidates are held against it."""
import json

import numpy as np
import pytest

import aldic_b200 as A
from aldic_b200 import synth_gpu

pytestmark = pytest.mark.gpu


def _entry(M, N, w, step, r, flat=False):
    p = synth_gpu.field_pair(6, M=M, N=N, umax=0.5 * r, gmax=0.02)
    c = A.Context(0)
    try:
        for slot, im in enumerate((p.ref, p.deff)):
            im = im.clone()
            if flat:
                im.view(N, M)[:, :M // 4] = 0
                im.view(N, M)[N // 2:N // 2 + 60, M // 2:M // 2 + 60] = 0
            c.load_image_raw(slot, im, [1, M], [1, N], want_stats=False, shape=(M, N))
        plain = c.integer_search([r, r], [1, M], [1, N], w, step)
        c.set_option(A.OPT_AUTOTUNE, 1)
        for _ in range(2):  # tuned, then by the kept choice
            got = c.integer_search([r, r], [1, M], [1, N], w, step)
            for k in ("u", "v"):
                assert np.array_equal(got[k], plain[k], equal_nan=True)
        rep = c.tuning_report()
    finally:
        c.close()
    assert len(rep) == 1
    return rep.popitem()[1]


@pytest.mark.parametrize("M,N,w,step,r,kernel,others", [
    (330, 300, 30, 16, 10, "fft", {"tile24", "tile16", "direct"}),
    (420, 431, 20, 5, 4, "fft", {"direct"}),       # a pair without a tile kernel
    (400, 300, 40, 90, 5, "direct", {"direct"}),   # too few subsets for the tables
])
def test_the_choice_by_size_is_reported(M, N, w, step, r, kernel, others):
    e = _entry(M, N, w, step, r)
    assert e["by_size"]["kernel"] == kernel and e["by_size"]["ms"] > 0
    assert set(e["ms"]) == others and all(t > 0 for t in e["ms"].values())
    names = {"by_size": kernel, "tile24": "tile", "tile16": "tile", "direct": "direct"}
    assert e["choice"]["kernel"] == names[e["choice"]["search"]]
    times = dict(e["ms"], by_size=e["by_size"]["ms"])
    assert times[e["choice"]["search"]] <= min(times.values()) + 1e-4  # as printed


def test_less_exact_candidates_do_not_win():
    """FP32 sums find spurious maxima in windows of one value; the transforms do not (test_gpu_search_flat.py)."""
    e = _entry(420, 400, 40, 10, 30, flat=True)
    assert e["by_size"]["kernel"] == "fft" and e["choice"]["search"] == "by_size"
    assert e["ms"]["direct"] < 0
    json.dumps(e)
