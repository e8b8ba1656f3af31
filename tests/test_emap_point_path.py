"""GPU: where the direct e-map forms no node sums it is the point-by-point path with its own cut,
whatever turned them off: the same bits as for a table that has no smooth form (at one exact radius,
which node radius 0 leaves where node sums have it).

The other table differs from AutoGrid's in one entry (60 A) that no atom is far enough to meet."""
import ctypes

import numpy as np
import pytest

import fastgrid_b200 as fg

pytestmark = pytest.mark.gpu


def _inputs():
    """Atoms about the grid and 38 A beside it, enough pairs and extent for node sums."""
    rng = np.random.default_rng(8)
    near = rng.normal(0, 5, (900, 3))
    far = rng.uniform(-3, 3, (200, 3)) + [38, 0, 0]
    xyz = np.concatenate([np.clip(near, -9, 9), far])
    xyzw = np.concatenate([xyz, rng.normal(0, 0.03, (len(xyz), 1))], axis=1)
    eps = fg.ddd_table()
    other = eps.copy()
    other[6000] *= 1.00001
    return fg.Grid(97, 101, 103, 0.1), xyzw, eps, other


def test_node_radius_zero():
    g, xyzw, eps, other = _inputs()
    ctx = fg.Context(0)
    ctx.tune(fg.AG_TUNE_EMAP_RNEAR, 11.75)
    try:
        want = ctx.emap(g, xyzw, other)
        assert not np.array_equal(ctx.emap(g, xyzw, eps), want)  # node sums
        ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 0)
        assert np.array_equal(ctx.emap(g, xyzw, eps), want)
        assert np.array_equal(ctx.emap(g, xyzw, other), want)
    finally:
        ctx.close()


def test_plain_mode():
    g, xyzw, eps, other = _inputs()
    ctx = fg.Context(0)
    ctx.tune(fg.AG_TUNE_EMAP_RNEAR, 11.75)
    try:
        want = ctx.emap(g, xyzw, other, mode=fg.AG_EMAP_PLAIN)
        assert np.array_equal(ctx.emap(g, xyzw, eps, mode=fg.AG_EMAP_PLAIN), want)
        kahan = ctx.emap(g, xyzw, eps)  # the mode is the call's own
        assert not np.array_equal(kahan, want)
        assert np.array_equal(ctx.emap(g, xyzw, eps), kahan)
    finally:
        ctx.close()


def test_node_radius_set_after_the_upload():
    g, xyzw, eps, other = _inputs()
    xyzw, eps = np.ascontiguousarray(xyzw), np.ascontiguousarray(eps)
    rec = fg.Receptor()
    rec.n_atoms = len(xyzw)
    rec.xyzw = xyzw.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    ctx = fg.Context(0)
    ctx.tune(fg.AG_TUNE_EMAP_RNEAR, 11.75)
    try:
        want = ctx.emap(g, xyzw, other)
        nodes = ctx.emap(g, xyzw, eps)
        ctx.upload(g, rec, None, eps.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        maps = np.empty(2 * want.size, dtype=np.float32)
        for radius, expect in ((0, want), (24, nodes), (0, want)):
            ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, radius)
            ctx.compute(fg.AG_WORK_EMAP)
            ctx.download(maps)
            assert np.array_equal(maps[:expect.size], expect.ravel()), radius
    finally:
        ctx.close()
