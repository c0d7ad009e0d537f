"""Device memory of the integer search: only what the chosen kernel reads, and the direct kernel, which needs
none beyond the integral images, where there is no memory for another's tables."""
import numpy as np
import pytest
import torch

import aldic_b200 as A
from aldic_b200 import synth_gpu

pytestmark = pytest.mark.gpu


def _load(c, M, N, seed=3):
    p = synth_gpu.field_pair(seed, M=M, N=N, umax=3.0, gmax=0.02)
    for slot, im in enumerate((p.ref, p.deff)):
        c.load_image_raw(slot, im, [1, M], [1, N], want_stats=False, shape=(M, N))
    c.synchronize()


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _search(c, M, N, r, w, step):
    return c.integer_search([r, r], [1, M], [1, N], w, step)


@pytest.mark.parametrize("w,step,r,tables", [
    (40, 200, 5, False),   # 81 subsets of a pair without a tile kernel: the direct kernel
    (32, 24, 20, True),    # transforms
])
def test_bytes_of_the_chosen_kernel(w, step, r, tables):
    M = N = 2048
    other = A.Context(0)  # the kernels' code is loaded before the count
    c = A.Context(0)
    try:
        _load(other, M, N)
        _search(other, M, N, r, w, step)
        _load(c, M, N)
        torch.cuda.empty_cache()
        before = _free()
        _search(c, M, N, r, w, step)
        taken = before - _free()
        images = 2 * 8 * (M + 1) * (N + 1)
        # the tile sums (4 MB) and the outputs' staging (1 MB), in blocks of 2 MB
        assert images <= taken <= images + (12 << 20) + (150 << 20 if tables else 0), taken
        assert not tables or taken > images + (40 << 20)
    finally:
        c.close()
        other.close()


def test_direct_kernel_without_memory_for_tables():
    M = N = 3000
    w, step, r = 32, 24, 6
    c = A.Context(0)
    try:
        _load(c, M, N)
        want = _search(c, M, N, r, w, step)
        n0 = c.launches
        _search(c, M, N, r, w, step)
        by_tables = c.launches - n0
        c.close()
        c = A.Context(0)
        _load(c, M, N)
        c.set_option(A.OPT_SEARCH_IMPL, 2)
        n0 = c.launches
        direct = _search(c, M, N, r, w, step)
        by_direct = c.launches - n0
        assert by_direct < by_tables
        c.set_option(A.OPT_SEARCH_IMPL, 0)
        torch.cuda.empty_cache()
        hog = torch.empty(_free() - (64 << 20), dtype=torch.uint8, device="cuda")  # the tables take 100 MB
        n0 = c.launches
        got = _search(c, M, N, r, w, step)
        assert c.launches - n0 == by_direct
        del hog
        torch.cuda.empty_cache()
        n0 = c.launches
        again = _search(c, M, N, r, w, step)
        assert c.launches - n0 == by_tables
        for k in ("x", "y", "u", "v", "phi"):
            assert np.array_equal(got[k], direct[k], equal_nan=True)
            assert np.array_equal(again[k], want[k], equal_nan=True)
    finally:
        c.close()
