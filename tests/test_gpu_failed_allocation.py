"""A call whose buffers do not fit the device's memory fails with an error and leaves the context usable: no
capacity or pointer of a freed buffer is kept, and the error is reported once."""
import numpy as np
import pytest
import torch

import aldic_b200 as A
from aldic_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture()
def hog():
    """Takes the device's memory but for the number of bytes it is called with."""
    held = []

    def take(left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda"))

    yield take
    held.clear()
    torch.cuda.empty_cache()


def _frame(c, sc):
    M, N = sc.ref.shape
    c.load_image_raw(0, sc.ref, [1, M], [1, N])
    c.load_image_raw(1, sc.deff, [1, M], [1, N])
    c.compute_gradients()


def _solve(c, n):
    xy = np.stack([np.tile(np.arange(60.0, 160.0, 10), n // 10 + 1)[:n], np.full(n, 90.0)], 1)
    return c.local_icgn(1, xy, np.zeros(2 * n), 20, 1e-3)


def test_scratch(hog):
    sc = synth.temporal_affine(M=220, N=200, n_speckles=900, u=0.4, v=-0.3)
    c = A.Context(0)
    try:
        _frame(c, sc)
        want = _solve(c, 100)
        hog(256 << 20)
        with pytest.raises(A.AldicError, match="memory"):
            _solve(c, 1_500_000)  # 0.9 GB
        for _ in range(2):
            got = _solve(c, 100)  # less than the scratch held before the failure
            assert np.array_equal(got["U"], want["U"]) and np.array_equal(got["conv"], want["conv"])
    finally:
        c.close()


def test_frame(hog):
    sc = synth.temporal_affine(M=220, N=200, n_speckles=900, u=0.4, v=-0.3)
    c = A.Context(0)
    try:
        _frame(c, sc)
        want = _solve(c, 100)
        hog(128 << 20)
        with pytest.raises(A.AldicError, match="memory"):
            c.load_image_raw(0, np.zeros((9000, 8000), np.uint8, order="F"), [1, 9000], [1, 8000])
        with pytest.raises(A.AldicError):
            _solve(c, 100)  # the former frame is gone
        with pytest.raises(A.AldicError):
            c.compute_gradients()
        _frame(c, sc)
        got = _solve(c, 100)
        assert np.array_equal(got["U"], want["U"]) and np.array_equal(got["conv"], want["conv"])
    finally:
        c.close()
