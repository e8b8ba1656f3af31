"""The direct e-map's node sums: atoms far from a CTA box enter through 5 x 5 x 5
Chebyshev nodes of the box instead of point by point.

CPU: a numpy restatement of the interpolation and of the dielectric's smooth form keeps the
errors that the kernel's rule relies on.  GPU: the node sums against the point-by-point path
(AG_TUNE_EMAP_NODE_RADIUS 0) and the FP64 oracle.
"""
import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

from conftest import E_TOL

LAMBDA, A, C = 0.3153767175, 7.7839, 66.57180475 / 78.4
NODES = np.cos((2 * np.arange(5) + 1) * np.pi / 10)


def _weights(t):
    w = np.ones((len(t), 5))
    for j in range(5):
        for m in range(5):
            if m != j:
                w[:, j] *= (t - NODES[m]) / (NODES[j] - NODES[m])
    return w


@pytest.mark.parametrize("half", [(2.81, 1.31, 2.81), (2.81, 2.81, 2.81), (0.4, 2.9, 2.9), (7.5, 3.5, 7.5)])
@pytest.mark.parametrize("ddd", [True, False])
def test_interpolation_error_at_the_least_distance(half, ddd):
    """At the least distance the kernel allows (8.5 half-widths and 24 A, or 9.5 half-widths for
    the constant dielectric), the interpolated term of one atom is within 4e-6 (1.3e-6) of the
    term, for directions along faces, edges and corners."""
    rng = np.random.default_rng(1)
    R = max(8.5 * max(half), 24.0) if ddd else 9.5 * max(half)
    axis = np.linspace(-1, 1, 9)
    W = _weights(axis)
    bound = 4e-6 if ddd else 1.3e-6
    for _ in range(150):
        d = rng.standard_normal(3) * (rng.random(3) > 0.3)
        if not d.any():
            continue
        d /= np.linalg.norm(d)
        a = np.where(d == 0, rng.uniform(-1, 1, 3), np.sign(d)) * half + R * d

        def f(x, y, z):
            r = np.sqrt((x[:, None, None] - a[0]) ** 2 + (y[:, None] - a[1]) ** 2 + (z - a[2]) ** 2)
            E = np.exp(-LAMBDA * (r - 0.005)) if ddd else 0 * r
            return (1 + E * ((A + C) + C * (A + C) * E)) / r

        F = f(*(NODES * h for h in half))
        got = np.einsum("xi,yj,zk,ijk->xyz", W, W, W, F)
        want = f(*(axis * h for h in half))
        assert (np.abs(got / want - 1) < bound).all()


def test_smooth_dielectric_is_the_table_between_its_steps():
    """From 24 A on the smooth form is the table at mid-bin: within 1e-9 of 332 / eps there, so
    within half a step (7.2e-6 of the value at 24 A, 2.8e-6 at 27 A) of the table's entry."""
    t = fg.ddd_table()
    b = np.arange(2400, 8191)
    r = (b + 0.5) / 100
    E = np.exp(-LAMBDA * (r - 0.005))
    smooth = 332.0 / 78.4 * (1 + E * ((A + C) + C * (A + C) * E))
    assert (np.abs(smooth / t[b] - 1) < 1e-9).all()
    step = np.abs(t[b + 1] - t[b]) / t[b]
    assert 0.5 * step[0] < 7.3e-6 and 0.5 * step[300] < 2.9e-6


FAR_NODES = np.cos((2 * np.arange(4) + 1) * np.pi / 8)


@pytest.mark.parametrize("half", [(2.81, 1.31, 2.81), (2.81, 2.81, 2.81), (0.4, 2.9, 2.9), (4.5, 2.1, 4.5)])
def test_far_node_error_at_the_least_distance(half):
    """From 57 A and 17.5 half-widths on: four nodes per axis and the saturated dielectric, within
    2.2e-6 (interpolation) and 1.4e-7 (the dielectric's part left out) of a term."""
    rng = np.random.default_rng(2)
    R = max(17.5 * max(half), 57.0)
    axis = np.linspace(-1, 1, 9)
    W = np.ones((9, 4))
    for j in range(4):
        for m in range(4):
            if m != j:
                W[:, j] *= (axis - FAR_NODES[m]) / (FAR_NODES[j] - FAR_NODES[m])
    for _ in range(150):
        d = rng.standard_normal(3) * (rng.random(3) > 0.3)
        if not d.any():
            continue
        d /= np.linalg.norm(d)
        a = np.where(d == 0, rng.uniform(-1, 1, 3), np.sign(d)) * half + R * d

        def r(x, y, z):
            return np.sqrt((x[:, None, None] - a[0]) ** 2 + (y[:, None] - a[1]) ** 2 + (z - a[2]) ** 2)

        got = np.einsum("xi,yj,zk,ijk->xyz", W, W, W, 1 / r(*(FAR_NODES * h for h in half)))
        want = r(*(axis * h for h in half))
        E = np.exp(-LAMBDA * (want - 0.005))
        assert (np.abs(got * want - 1) < 2.2e-6).all()
        assert (E * ((A + C) + C * (A + C) * E) < 1.4e-7).all()


def _atoms(rng, n, spread):
    """Atoms around the grid and on shells out to 120 A, some far outside."""
    inner = rng.normal(0, spread, (n, 3))
    shell = rng.standard_normal((n, 3))
    shell *= (rng.uniform(18, 120, (n, 1)) / np.linalg.norm(shell, axis=1, keepdims=True))
    xyz = np.concatenate([inner, shell, [[900.0, -700.0, 20.0]]])
    return np.concatenate([xyz, rng.normal(0, 0.03, (len(xyz), 1))], axis=1)


# Shapes: full and ragged tiles, one-point and one-row grids, a last odd x column, grids thinner
# than a tile; spacings whose boxes reach the radius rule's both sides; atom counts around a tile.
GRIDS = [(33, 45, 29, 0.375), (41, 9, 17, 0.375), (1, 1, 1, 0.375), (129, 1, 1, 0.375), (1, 70, 3, 0.375),
         (24, 23, 22, 1.0), (45, 37, 31, 2.0), (40, 40, 40, 0.1)]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,h", GRIDS)
@pytest.mark.parametrize("n", [1, 128, 1100])
def test_node_sums_match_point_sums_and_oracle(nx, ny, nz, h, n):
    """Against the point-by-point path: each far term may differ by its interpolation error
    (4e-6), half a table step (7.3e-6 at 24 A, 2.9e-6 at 27 A) and FP32 rounding (1e-6), so the
    sums by as much of the sum of the terms' magnitudes."""
    rng = np.random.default_rng(nx * 1000 + n)
    xyzw = _atoms(rng, n, 9.0)
    g = fg.Grid(nx, ny, nz, h)
    ctx = fg.Context(0)
    try:
        for eps in (fg.ddd_table(), None):
            ref = oracle.emap(g, xyzw, eps)
            mag = oracle.emap(g, np.abs(xyzw) * [0, 0, 0, 1] + xyzw * [1, 1, 1, 0], eps)
            ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 0)
            point = ctx.emap(g, xyzw, eps)
            for radius, tol in ((27, 7.9e-6), (24, 12.3e-6)):
                ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, radius)
                got = ctx.emap(g, xyzw, eps)
                assert (np.abs(got - point.astype(np.float64)) <= tol * mag + 1e-7).all()
                assert np.abs(got - ref).max() <= E_TOL
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,h", [(33, 45, 29, 0.375), (41, 9, 17, 0.375), (129, 1, 1, 0.375),
                                        (24, 23, 22, 0.6), (24, 23, 22, 0.7), (45, 37, 31, 1.0)])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1100])
@pytest.mark.parametrize("mixed", [False, True])
def test_far_nodes_match_point_sums_and_oracle(nx, ny, nz, h, n, mixed):
    """Atoms beyond 57 A of every box alone (odd and even counts around a tile), and in one list with
    nearer ones of every class.  Alone, a term may differ by its interpolation error (2.2e-6 far;
    4e-6 where wide boxes keep five nodes), the dielectric left out and FP32 rounding (1e-6);
    mixed, by the node sums' own 12.3e-6."""
    rng = np.random.default_rng(nx + n)
    ends = np.array([nx, ny, nz]) * h / 2
    d = rng.standard_normal((n, 3))
    d /= np.abs(d).max(axis=1, keepdims=True)
    xyz = d * (ends.max() + rng.uniform(58, 140, (n, 1)))  # one coordinate past the grid by that much
    xyzw = np.concatenate([xyz, rng.normal(0, 0.03, (n, 1))], axis=1)
    if mixed:
        xyzw = np.concatenate([xyzw, _atoms(rng, 150, 9.0)])
        xyzw = xyzw[rng.permutation(len(xyzw))]
    g = fg.Grid(nx, ny, nz, h)
    eps = fg.ddd_table()
    ref = oracle.emap(g, xyzw, eps)
    mag = oracle.emap(g, np.abs(xyzw) * [0, 0, 0, 1] + xyzw * [1, 1, 1, 0], eps)
    ctx = fg.Context(0)
    try:
        ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 0)
        point = ctx.emap(g, xyzw, eps)
        ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 24)
        got = ctx.emap(g, xyzw, eps)
        tol = 12.3e-6 if mixed else 5.2e-6
        assert (np.abs(got - point.astype(np.float64)) <= tol * mag + 1e-7).all()
        assert np.abs(got - ref).max() <= E_TOL
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,h", GRIDS + [(20, 300, 301, 0.375)])
def test_allocation_free_call_matches_oracle(nx, ny, nz, h):
    """ag_emap_noalloc on the same shapes, both dielectrics and a table that is not AutoGrid's
    (sampled points on the largest, whose tiles are all ragged)."""
    import ctypes

    import torch

    rng = np.random.default_rng(nx + ny)
    xyzw = _atoms(rng, 500, 9.0)
    g = fg.Grid(nx, ny, nz, h)
    idx = np.unique(rng.integers(0, nx * ny * nz, 3000))
    d_xyzw = torch.from_numpy(xyzw).cuda()
    for eps in (fg.ddd_table(), None, fg.ddd_table() * 0.5):
        d_eps = None if eps is None else torch.from_numpy(eps).float().cuda()
        out = torch.full((nx * ny * nz,), float("nan"), device="cuda")
        rc = fg.lib().ag_emap_noalloc(ctypes.byref(g), len(xyzw), d_xyzw.data_ptr(),
                                      None if eps is None else d_eps.data_ptr(), out.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)
        assert rc == fg.AG_OK, fg.lib().ag_last_error()
        want = oracle.emap_points(g, xyzw, eps, idx)
        assert np.abs(out.cpu().numpy()[idx] - want).max() <= E_TOL


@pytest.mark.gpu
def test_other_tables_are_summed_point_by_point():
    """A table that is not AutoGrid's function keeps the point path: the same bits as with the
    node sums turned off."""
    rng = np.random.default_rng(5)
    xyzw = _atoms(rng, 600, 9.0)
    g = fg.Grid(33, 29, 31, 0.375)
    eps = fg.ddd_table()
    ctx = fg.Context(0)
    try:
        for table in (eps * 0.5, np.where(np.arange(8192) == 7000, eps * 1.001, eps)):
            on = ctx.emap(g, xyzw, table)
            assert np.abs(on - oracle.emap(g, xyzw, table)).max() <= E_TOL
            ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 0)
            assert np.array_equal(on, ctx.emap(g, xyzw, table))
            ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 24)
        with pytest.raises(fg.AgError):
            ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 10)
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [970, 971])
def test_both_sides_of_the_few_pairs_rule(n):
    """970 and 971 atoms on 101^3 points lie on either side of 1e9 pairs, below which no node sums are
    formed: both match the oracle, and a node radius set by hand (node sums on either side) within
    the node sums' 12.3e-6 of the terms' magnitudes."""
    rng = np.random.default_rng(3)
    xyzw = _atoms(rng, 485, 9.0)[:n]
    if len(xyzw) < n:
        xyzw = np.concatenate([xyzw, _atoms(rng, 1, 9.0)[:n - len(xyzw)]])
    g = fg.Grid(101, 101, 101, 0.375)
    idx = np.unique(rng.integers(0, 101 ** 3, 3000))
    eps = fg.ddd_table()
    want = oracle.emap_points(g, xyzw, eps, idx)
    mag = oracle.emap_points(g, np.abs(xyzw) * [0, 0, 0, 1] + xyzw * [1, 1, 1, 0], eps, idx)
    ctx = fg.Context(0)
    try:
        default = ctx.emap(g, xyzw, eps).ravel()[idx].astype(np.float64)
        ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 24)
        nodes = ctx.emap(g, xyzw, eps).ravel()[idx]
    finally:
        ctx.close()
    assert len(xyzw) == n
    assert np.abs(default - want).max() <= E_TOL
    assert (np.abs(nodes - default) <= 12.3e-6 * mag + 1e-7).all()
