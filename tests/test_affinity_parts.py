"""GPU: the two-point affinity kernel's plan of a pass.

Ligand type sets whose passes sit at the edges of the plan: rows of 4, 8, 12 and 16 columns (maps
plus the desolvation column) just full and just over, no ligand map, no H-bonding probe, only
H-bonding probes, more than four of them (several passes), and sets whose maps share columns for
every receptor type, for all but the donors, or never.  Every map against the FP64 oracle with the
parity tests' tolerances, and against the one-point kernel.
"""
import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

from conftest import AFF_ABS, aff_tol, chdir

pytestmark = pytest.mark.gpu

SETS = ["C", "HD", "A C N", "A C HD N", "C N OA S F Cl Br", "A C HD N OA SA S", "A C HD N NA OA SA S",
        "C A N S F Cl Br I P Zn Fe", "C A N S F Cl Br I P Zn Fe Mg", "C A N S HD F Cl Br I P Zn Fe Mg Ca",
        "HD HS NA NS OA OS SA", "A C HD HS N NA NS OA OS SA S F Cl Br"]


@pytest.mark.parametrize("types", SETS)
@pytest.mark.parametrize("npts", [8, 22])
def test_type_sets_match_oracle(tmp_path, types, npts):
    fg.synth_write(str(tmp_path), "t", n_atoms=700, semi_axes=(13, 12, 11), npts=npts, seed=41, ligand_types=types)
    with chdir(str(tmp_path)):
        p = fg.Problem("t.gpf", log="t.glg")
    want, wantd = oracle.affinity(p.grid, p.receptor, p.params)
    got = {}
    for kernel in (2, 1):
        ctx = fg.Context(0)
        try:
            ctx.tune(fg.AG_TUNE_AFFINITY_KERNEL, kernel)
            got[kernel] = ctx.affinity(p.grid, p.receptor, p.params, p.n_maps)
        finally:
            ctx.close()
        maps, d = got[kernel]
        for m in range(p.n_maps):
            assert (np.abs(maps[m] - want[m]) <= aff_tol(want[m])).all(), (kernel, m)
        assert np.abs(d - wantd).max() <= AFF_ABS
    for m in range(p.n_maps):
        assert (np.abs(got[1][0][m].astype(np.float64) - got[2][0][m]) <= 2 * aff_tol(want[m])).all()


@pytest.mark.parametrize("kernel", [2, 1])
def test_without_ligand_maps(tmp_path, kernel):
    """No ligand map at all: the desolvation map alone."""
    fg.synth_write(str(tmp_path), "t", n_atoms=500, semi_axes=(12, 11, 10), npts=14, seed=42, ligand_types="C")
    with chdir(str(tmp_path)):
        p = fg.Problem("t.gpf", log="t.glg")
    par = fg.AffinityParams.from_buffer_copy(p.params)
    par.n_maps = 0
    ctx = fg.Context(0)
    try:
        ctx.tune(fg.AG_TUNE_AFFINITY_KERNEL, kernel)
        maps, d = ctx.affinity(p.grid, p.receptor, par, 0)
    finally:
        ctx.close()
    assert maps.shape[0] == 0
    assert np.abs(d - oracle.affinity(p.grid, p.receptor, p.params)[1]).max() <= AFF_ABS
