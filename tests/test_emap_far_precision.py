"""The node sums' precision wherever the grid lies to the receptor.

GPU: the relative 2-norm error against the FP64 oracle with node sums is no larger than that of
summing every atom at every point with exact bins to 11 A, for a grid inside the receptor, over its
surface and 12, 24 and 54 A beside it, and for both dielectrics.  The two are independent FP32
evaluations of the same sums, whose 2-norms over 4,000 points differ by a few percent by chance:
10 % are allowed (the receptors, grids and points are fixed).
CPU: nodes on multiples of 0.005 A stay distinct and interpolate as well as the Chebyshev ones.
"""
import ctypes

import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

LAMBDA, A, C = 0.3153767175, 7.7839, 66.57180475 / 78.4


def _offset_receptor(n, offset):
    a = fg.surrogate_receptor(3, n).copy()
    a[:, :3] += np.array([1, 0.6, 0.3]) / np.linalg.norm([1, 0.6, 0.3]) * offset
    return a


def _noalloc(g, xyzw, eps):
    import torch

    d_xyzw = torch.from_numpy(np.ascontiguousarray(xyzw)).cuda()
    d_eps = None if eps is None else torch.from_numpy(eps).float().cuda()
    out = torch.empty(g.nx * g.ny * g.nz, device="cuda")
    rc = fg.lib().ag_emap_noalloc(ctypes.byref(g), len(xyzw), d_xyzw.data_ptr(),
                                  None if d_eps is None else d_eps.data_ptr(), out.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == fg.AG_OK, fg.lib().ag_last_error()
    return out.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("n,points,offset", [(20000, 41, 0), (20000, 41, 43), (20000, 41, 63), (20000, 41, 75),
                                             (20000, 41, 105), (8000, 51, 45), (8000, 101, 0)])
@pytest.mark.parametrize("ddd", [True, False])
def test_no_less_precise_than_point_sums(n, points, offset, ddd):
    xyzw = _offset_receptor(n, offset)
    eps = fg.ddd_table() if ddd else None
    g = fg.Grid(points, points, points, 0.375)
    idx = np.unique(np.random.default_rng(n + offset).integers(0, points ** 3, 4000))
    want = oracle.emap_points(g, xyzw, eps, idx)

    def err(e):
        return np.linalg.norm(e.ravel()[idx].astype(np.float64) - want)

    ctx = fg.Context(0)
    try:
        nodes = err(ctx.emap(g, xyzw, eps))
        ctx.tune(fg.AG_TUNE_EMAP_NODE_RADIUS, 0)
        ctx.tune(fg.AG_TUNE_EMAP_RNEAR, 11)
        point = err(ctx.emap(g, xyzw, eps))
    finally:
        ctx.close()
    assert nodes <= 1.1 * point, (nodes / point, point / np.linalg.norm(want))
    noalloc = err(_noalloc(g, xyzw, eps))
    assert noalloc <= 1.1 * point, (noalloc / point, point / np.linalg.norm(want))


@pytest.mark.parametrize("ddd", [True, False])
@pytest.mark.parametrize("half", [(2.8225, 1.3225, 2.8225), (2.8225, 2.8225, 2.8225), (0.01, 0.3, 2.9),
                                  (0.385, 0.01, 0.01), (7.51, 3.51, 7.51)])
def test_snapped_nodes_interpolate_as_chebyshev_nodes(half, ddd):
    """Half extents as the boxes have them (0.01 A wider than the points).  The bounds are those of
    the Chebyshev nodes at the least distances, 4e-6 and 1.3e-6 of a term."""
    rng = np.random.default_rng(1)
    cheb = np.cos((2 * np.arange(5) + 1) * np.pi / 10)
    nodes = [np.rint(2 * cheb * 100 * h) / 200 for h in half]
    assert all(len(set(x)) == 5 for x in nodes)
    axes = [np.linspace(-h, h, 9) for h in half]
    W = []
    for x, t in zip(nodes, axes):
        w = np.ones((9, 5))
        for j in range(5):
            for m in range(5):
                if m != j:
                    w[:, j] *= (t - x[m]) / (x[j] - x[m])
        W.append(w)
    R, bound = (max(8.5 * max(half), 24.0), 4e-6) if ddd else (9.5 * max(half), 1.3e-6)
    for _ in range(150):
        d = rng.standard_normal(3) * (rng.random(3) > 0.3)
        if not d.any():
            continue
        d /= np.linalg.norm(d)
        a = np.where(d == 0, rng.uniform(-1, 1, 3), np.sign(d)) * half + R * d

        def f(x, y, z):
            r = np.sqrt((x[:, None, None] - a[0]) ** 2 + (y[:, None] - a[1]) ** 2 + (z - a[2]) ** 2)
            e = np.exp(-LAMBDA * (r - 0.005)) if ddd else 0 * r
            return (1 + e * ((A + C) + C * (A + C) * e)) / r

        got = np.einsum("xi,yj,zk,ijk->xyz", *W, f(*nodes))
        assert (np.abs(got / f(*axes) - 1) < bound).all()
