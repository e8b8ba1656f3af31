"""GPU: batches take their context's e-map options, and mix jobs of different probe sets."""
import numpy as np
import pytest

import fastgrid_b200 as fg
import oracle

from conftest import AFF_ABS, E_TOL, aff_tol, chdir

pytestmark = pytest.mark.gpu

# One, two and four affinity passes in one launch, rows of 4, 8, 12 and 16 columns.
JOBS = [(1500, 41, "C HD"), (900, 25, "A C HD HS N NA NS OA OS SA S F Cl Br"), (2500, 31, "A C HD N OA SA"),
        (700, 33, "C"), (1200, 27, "HD HS NA NS OA OS SA C A N S F")]


def _problems(tmp, jobs):
    out = []
    for k, (n, g, types) in enumerate(jobs):
        r = 20.0 * (n / 2000.0) ** (1 / 3)
        fg.synth_write(str(tmp), f"b{k}", n_atoms=n, semi_axes=(r, r, r), npts=g - 1, seed=60 + k, ligand_types=types)
        with chdir(str(tmp)):
            out.append(fg.Problem(f"b{k}.gpf", log=f"b{k}.glg"))
    return out


def test_mixed_probe_sets_match_oracle(tmp_path):
    probs = _problems(tmp_path, JOBS)
    ctx = fg.Context(0)
    b = fg.Batch(ctx, probs)
    first = None
    for _ in range(3):
        b.compute()
        got = [b.maps(i) for i in range(len(probs))]
        if first is None:
            first = got
            continue
        for i in range(len(probs)):
            assert np.array_equal(got[i], first[i]), f"graph replay differs for job {i}"
    for i, p in enumerate(probs):
        flat = first[i].reshape(p.n_maps + 2, -1)
        maps, d = oracle.affinity(p.grid, p.receptor, p.params)
        for m in range(p.n_maps):
            assert (np.abs(flat[m] - maps[m]) <= aff_tol(maps[m])).all(), (i, m)
        assert np.abs(flat[p.n_maps] - oracle.emap(p.grid, p.xyzw(), p.inv_eps())).max() <= E_TOL
        assert np.abs(flat[p.n_maps + 1] - d).max() <= AFF_ABS
    b.close()
    ctx.close()


def _batch_emap(p, knobs):
    ctx = fg.Context(0)
    for k, v in knobs:
        ctx.tune(k, v)
    b = fg.Batch(ctx, [p])
    b.compute()
    e = b.maps(0).reshape(p.n_maps + 2, -1)[p.n_maps].copy()
    b.close()
    ctx.close()
    return e


@pytest.mark.parametrize("knob,value", [(fg.AG_TUNE_EMAP_NODE_RADIUS, 0), (fg.AG_TUNE_EMAP_NODE_RADIUS, 30),
                                        (fg.AG_TUNE_EMAP_RNEAR, 14), (fg.AG_TUNE_EMAP_PACKED_TABLE, 0)])
def test_batch_takes_the_contexts_emap_options(tmp_path, knob, value):
    """Each option changes some of the map's last bits, and keeps it within tolerance."""
    p = _problems(tmp_path, [(20000, 45, "C HD")])[0]  # reaches far enough for node sums
    default, tuned = _batch_emap(p, []), _batch_emap(p, [(knob, value)])
    assert not np.array_equal(default, tuned)
    want = oracle.emap(p.grid, p.xyzw(), p.inv_eps())
    assert np.abs(tuned - want).max() <= E_TOL and np.abs(default - want).max() <= E_TOL


def test_batch_keeps_no_staged_inputs(tmp_path):
    """A job's staged inputs (about 400 KB) are not kept once it is on the device: the process grows by
    less than half of that per job (the host copies of the table and the boxes take some 80 KB)."""
    probs = _problems(tmp_path, [(2000, 31, "A C HD N OA SA")])

    def resident():
        return int(next(l for l in open("/proc/self/status") if l.startswith("VmRSS")).split()[1]) * 1024

    grown = []
    for _ in range(2):  # the first also loads code
        ctx = fg.Context(0)
        before = resident()
        b = fg.Batch(ctx, probs * 48)
        grown.append(resident() - before)
        b.close()
        ctx.close()
    assert grown[1] < 48 * 200e3


def test_batch_counts_its_kernels(tmp_path):
    """Node radii, e-map, cell list, slot maps' zeroing and affinity pass; a receptor of more than 8,192
    atoms takes four kernels for its cell list."""
    probs = _problems(tmp_path, [(1000, 25, "C HD"), (9000, 25, "C HD"), (1000, 25, "C")])
    ctx = fg.Context(0)
    count = []
    for p in probs:
        b = fg.Batch(ctx, [p])
        for _ in range(2):
            before = ctx.launches
            b.compute()
            count.append(ctx.launches - before)
        b.close()
    ctx.close()
    assert count == [5, 5, 8, 8, 4, 4]
