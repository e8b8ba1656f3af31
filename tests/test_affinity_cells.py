"""GPU: the affinity pass on widely spaced grids."""
import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

from conftest import AFF_ABS, aff_tol, chdir

pytestmark = pytest.mark.gpu


def _problem(tmp_path):
    fg.synth_write(str(tmp_path), "t", n_atoms=400, semi_axes=(11, 10, 9), npts=14, seed=43, ligand_types="C HD OA")
    with chdir(str(tmp_path)):
        return fg.Problem("t.gpf", log="t.glg")


@pytest.mark.parametrize("kernel", [2, 1])
@pytest.mark.parametrize("nx,ny,nz,h", [(1025, 1025, 3, 200.0), (129, 129, 129, 1.0e9)])
def test_more_cells_than_keys_are_refused(tmp_path, kernel, nx, ny, nz, h):
    """25,602 x 25,602 x 52 cells of 8 A are 3e10, more than 32-bit keys; the other grid's do not even
    count in 32 bits along an axis."""
    p = _problem(tmp_path)
    ctx = fg.Context(0)
    try:
        ctx.tune(fg.AG_TUNE_AFFINITY_KERNEL, kernel)
        with pytest.raises(fg.AgError) as e:
            ctx.affinity(fg.Grid(nx, ny, nz, h), p.receptor, p.params, p.n_maps)
        assert e.value.code == fg.AG_E_INVALID
        maps, _ = ctx.affinity(p.grid, p.receptor, p.params, p.n_maps)  # the context goes on
        want, _ = oracle.affinity(p.grid, p.receptor, p.params)
        assert all((np.abs(maps[m] - want[m]) <= aff_tol(want[m])).all() for m in range(p.n_maps))
    finally:
        ctx.close()


@pytest.mark.parametrize("kernel", [2, 1])
@pytest.mark.parametrize("h", [0.9, 2.0])
def test_wide_spacings_match_oracle(tmp_path, kernel, h):
    p = _problem(tmp_path)
    g = fg.Grid(9, 7, 8, h)
    ctx = fg.Context(0)
    try:
        ctx.tune(fg.AG_TUNE_AFFINITY_KERNEL, kernel)
        maps, d = ctx.affinity(g, p.receptor, p.params, p.n_maps)
    finally:
        ctx.close()
    want, wantd = oracle.affinity(g, p.receptor, p.params)
    for m in range(p.n_maps):
        assert (np.abs(maps[m] - want[m]) <= aff_tol(want[m])).all()
    assert np.abs(d - wantd).max() <= AFF_ABS
