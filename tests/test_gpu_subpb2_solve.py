"""The global step's one-launch solve at the sizes where its form changes: meshes of one and of
several nodes per thread, a node with more neighbours than a matrix row keeps, and a solve of more
iterations than one launch runs.  Against the oracle's direct solve."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import aldic_b200

    c = aldic_b200.Context(0)
    yield c
    c.close()


def _grid(nx, ny, h=4.0):
    X, Y = np.meshgrid(5 + h * np.arange(nx), 7 + h * np.arange(ny), indexing="ij")
    C = np.stack([X.ravel(order="F"), Y.ravel(order="F")], 1)
    j, i = np.meshgrid(np.arange(ny - 1), np.arange(nx - 1), indexing="ij")
    a = (j * nx + i).ravel() + 1
    E = np.zeros((a.size, 8), np.int32)
    E[:, 0], E[:, 1], E[:, 2], E[:, 3] = a, a + 1, a + nx + 1, a + nx
    return C, E


def _fan(spokes):
    """spokes quads around one node, which then has 2 spokes + 1 neighbours (itself among them)."""
    t = 2 * np.pi * np.arange(2 * spokes) / (2 * spokes)
    r = np.where(np.arange(2 * spokes) % 2 == 0, 10.0, 14.0)
    C = np.concatenate([[[50.0, 50.0]], np.stack([50 + r * np.cos(t), 50 + r * np.sin(t)], 1)])
    E = np.zeros((spokes, 8), np.int32)
    for k in range(spokes):
        E[k, :4] = [1, 2 + 2 * k, 3 + 2 * k, 2 + (2 * k + 2) % (2 * spokes)]
    return C, E


def _case(mesh):
    C, E = mesh
    rng = np.random.default_rng(len(C))
    n = len(C)
    s = C / np.abs(C).max()
    U = np.stack([np.sin(3 * s[:, 0]) + s[:, 1], np.cos(2 * s[:, 1]) * s[:, 0]], 1) + rng.normal(0, 0.01, (n, 2))
    return C, E, U.ravel(), rng.normal(0, 0.01, 4 * n)


@pytest.mark.parametrize("mesh", ["one_node", "one_per_thread", "ragged", "several_per_thread", "fan15", "fan16", "fan40"])
def test_solve_forms(ctx, mesh):
    # the largest grid of CTAs covers 148 x 3 x 128 = 56 832 nodes; rows of up to 12 entries are
    # kept in registers and of up to 32 in the assembled matrix (a fan of 16 has 33)
    m = {"one_node": lambda: _grid(2, 2), "one_per_thread": lambda: _grid(120, 90), "ragged": lambda: _grid(131, 3),
         "several_per_thread": lambda: _grid(270, 260), "fan15": lambda: _fan(15), "fan16": lambda: _fan(16),
         "fan40": lambda: _fan(40)}[mesh]()
    C, E, U, F = _case(m)
    d = np.array([1, 2, len(C) - 1], np.int32) if len(C) > 100 else None
    got, (it, ok) = ctx.subpb2(C, E, 2, 0.3, 1e-2, U, F, dirichlet=d, info=True)
    ref = O.subpb2_quadtree(C, E, 2, 0.3, 1e-2, U, F, dirichlet=() if d is None else d)
    assert ok == 1 and it >= 1
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()


def test_solve_continues_over_launches(ctx):
    # a strip 2 nodes wide: the information travels one element an iteration, so the solve takes
    # at least as many iterations as the strip is long, more than the 4096 of one launch.  The
    # residual tolerance 1e-12 and the strip's conditioning (length^2 = 3e7) leave 1e-4 of the field.
    C, E = _grid(5200, 2)
    n = len(C)
    rng = np.random.default_rng(1)
    U, F = rng.normal(0, 1, 2 * n), rng.normal(0, 0.01, 4 * n)
    d = np.array([1, 5201], np.int32)
    got, (it, ok) = ctx.subpb2(C, E, 2, 1.0, 1e-9, U, F, dirichlet=d, info=True)
    ref = O.subpb2_quadtree(C, E, 2, 1.0, 1e-9, U, F, dirichlet=d)
    assert ok == 1 and it > 4096
    assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()
