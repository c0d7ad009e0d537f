"""The global step's solve at the sizes where its grid of CTAs changes: the last mesh with one node a thread
(148 x 3 x 128 = 56 832 nodes), the first with the wider grid, and one with more nodes than that grid has threads
(148 x 7 x 128 = 132 608).  Strips, which the oracle solves fast.  Against the oracle's direct solve, to
1e-9 of the field as in test_gpu_subpb2_solve.py."""
import numpy as np
import pytest

import oracle as O
from test_gpu_subpb2_solve import _case, _grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3552, 16), (3553, 16), (8400, 16)])
def test_grids_of_the_solve(nx, ny):
    import aldic_b200

    C, E, U, F = _case(_grid(nx, ny))
    d = np.array([1, 2, len(C) - 1], np.int32)
    c = aldic_b200.Context(0)
    try:
        got, (it, ok) = c.subpb2(C, E, 2, 0.3, 1e-2, U, F, dirichlet=d, info=True)
    finally:
        c.close()
    ref = O.subpb2_quadtree(C, E, 2, 0.3, 1e-2, U, F, dirichlet=d)
    assert ok == 1 and it >= 1
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
