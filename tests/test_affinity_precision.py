"""GPU: the two-point affinity kernel's sums are more exact than sums in cell order.

A point's FP32 sum is rounded at the size of its largest term from that term on.  The one-point
kernel takes the atoms cell by cell, so the largest term comes anywhere; the two-point kernel takes
them type by type, those with the largest energies at close contact last, so fewer terms follow it.
Sums that ignored the energies would differ by chance, by 1 to 2 % of the 2-norm per receptor; three
receptors together have to gain 5 %.
"""
import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

from conftest import chdir

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", ["C HD", "A C HD N OA SA", "A C HD N NA OA SA S F Cl"])
def test_large_terms_are_summed_last(tmp_path, types):
    err = {1: 0.0, 2: 0.0}
    for seed in (5, 6, 7):
        fg.synth_write(str(tmp_path), "t", n_atoms=3000, semi_axes=(24, 22, 20), npts=46, seed=seed,
                       ligand_types=types)
        with chdir(str(tmp_path)):
            p = fg.Problem("t.gpf", log="t.glg")
        want = oracle.affinity(p.grid, p.receptor, p.params)[0].reshape(p.n_maps, -1)
        norm = np.linalg.norm(want, axis=1)
        for kernel in err:
            ctx = fg.Context(0)
            try:
                ctx.tune(fg.AG_TUNE_AFFINITY_KERNEL, kernel)
                got = ctx.affinity(p.grid, p.receptor, p.params, p.n_maps)[0].reshape(p.n_maps, -1)
            finally:
                ctx.close()
            err[kernel] += (np.linalg.norm(got - want, axis=1) / norm).mean()
    assert err[2] <= 0.95 * err[1], err
