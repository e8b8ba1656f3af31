"""GPU: every point that a CTA of the direct e-map evaluates lies in the CTA's box, on which the
choice of each atom's arithmetic and the clamps of the table reads rely.

Atoms 20 A and more beyond the grid enter by table reads alone.  Each term is then within one
0.01 A step of the table (5.2e-5 of it at 20 A, where FP32 may take the neighbouring bin), FP32
rounding (1e-6) and the rounding of coordinates in a wide box (2^-23 of its extent, of 20 A) of
the oracle's, so a sum is within as much of the sum of its terms' magnitudes.
"""
import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

pytestmark = pytest.mark.gpu


def _check(nx, ny, nz, h, order):
    rng = np.random.default_rng(nx * 100 + ny)
    n = 600
    half = np.array([nx, ny, nz]) * h / 2
    xyz = rng.uniform(-1, 1, (n, 3)) * half
    axis = rng.integers(0, 3, n)
    xyz[np.arange(n), axis] = rng.choice([-1, 1], n) * (half[axis] + rng.uniform(20, 45, n))
    xyzw = np.concatenate([xyz, rng.normal(0, 0.3, (n, 1))], axis=1)
    g = fg.Grid(nx, ny, nz, h)
    eps = fg.ddd_table()
    ctx = fg.Context(0)
    try:
        ctx.tune(fg.AG_TUNE_EMAP_WARP_COMPACT, order)
        got = ctx.emap(g, xyzw, eps)
    finally:
        ctx.close()
    want = oracle.emap(g, xyzw, eps)
    mag = oracle.emap(g, np.abs(xyzw) * [0, 0, 0, 1] + xyzw * [1, 1, 1, 0], eps)
    tol = 5.3e-5 + 2.0 ** -23 * half.max() / 20
    assert (np.abs(got - want) <= tol * mag + 1e-7).all()


@pytest.mark.parametrize("nx,ny,nz", [(49, 53, 27), (33, 45, 33), (21, 45, 55), (37, 53, 25)])
@pytest.mark.parametrize("h", [0.375, 0.7])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_interleaved_columns_stay_in_one_box(nx, ny, nz, h, order):
    """Odd row and plane counts of the last, unpaired column leave the pairs after it at odd places
    of the item list."""
    _check(nx, ny, nz, h, order)


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (1, 3, 2), (9, 2, 1), (10, 5, 5), (23, 4, 4)])
@pytest.mark.parametrize("h", [2.0, 8.0, 27.0, 400.0])
def test_points_past_the_end_of_widely_spaced_rows(nx, ny, nz, h):
    """Rows are evaluated in whole eights: the points past the grid's end of a wide spacing lie far
    outside the box unless they are folded onto it."""
    _check(nx, ny, nz, h, 2)
