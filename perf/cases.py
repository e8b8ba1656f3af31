"""Timed cases of the grid-map engine, each through an entry point that a program calls.

A case names its path (`path`), its sizes and its options:

  job        a docking set-up: a parsed GPF job, the whole map set into host memory
             (Problem.compute; every call uploads the job's arrays and copies the maps back)
  resident   a job uploaded once and computed in device memory (Context.upload / compute): the
             whole map set, the affinity pass, the direct e-map or the surrogate e-map
  emap       the e-map seam with host arrays (Context.emap), as FastGrid's driver calls it
  noalloc    the e-map on the caller's own device buffers (ag_emap_noalloc)
  batch      many receptors in persistent kernels under one CUDA graph (Batch)
  net_grad   one forward and backward pass of the surrogate's corrector network

Receptors are the engine's seeded synthetic globules (a self-avoiding chain walk at protein
density, AutoDock types and clipped normal charges); grids are 0.375 A unless a case says
otherwise, odd and unequal along the axes where the entry point takes any shape.
"""
import ctypes
import os
import tempfile

import numpy as np
import torch

import fastgrid_b200 as fg

TYPES = {
    2: "C HD",
    6: "A C HD N OA SA",
    10: "A C HD N NA OA SA S F Cl",
    14: "A C HD HS N NA NS OA OS SA S F Cl Br",  # more than four H-bonding probes
}


# --- the cases ---------------------------------------------------------------------------------
def listed():
    return [
        # A fragment or a binding-site cut-out with two probe types: launches and host work count.
        dict(name="job_fragment", path="job", atoms=400, points=31, maps=2, diel=-0.1465),
        # A usual docking box around a small receptor (the small configuration of bench.py).
        dict(name="job_small", path="job", atoms=2000, points=61, maps=6, diel=-0.1465),
        # Blind docking over a large receptor (bench.py's default workload).
        dict(name="job_large", path="job", atoms=20000, points=161, maps=10, diel=-0.1465),
        # The constant dielectric, a finer grid and a box smaller than the receptor.
        dict(name="job_constant_dielectric", path="job", atoms=6000, points=93, maps=6, diel=40.0, spacing=0.25),
        # A conformer loop that keeps its maps on the device; a ragged box.
        dict(name="resident_map_set", path="resident", work="all", atoms=8000, nx=125, ny=97, nz=83, maps=6),
        # The affinity pass alone (other probes on a receptor whose e-map is known); a ragged box.
        dict(name="resident_affinity", path="resident", work="affinity", atoms=12000, nx=131, ny=119, nz=101, maps=10),
        # The e-map of a very large complex (the precision study's size).
        dict(name="resident_emap_complex", path="resident", work="emap", atoms=60000, nx=255, ny=255, nz=255, maps=0),
        # The learned far-field e-map on a held-out receptor's grid.
        dict(name="resident_surrogate", path="resident", work="surrogate", atoms=20000, nx=161, ny=161, nz=161, maps=0),
        # FastGrid's e-map seam: host arrays in, a host map out.
        dict(name="emap_host", path="emap", atoms=5000, nx=101, ny=87, nz=73),
        # A host with its own memory pool: device buffers in and out.
        dict(name="emap_noalloc", path="noalloc", atoms=3500, nx=121, ny=113, nz=89, diel=-0.1465),
        # A screening set of receptors of uneven sizes.
        dict(name="batch_uneven", path="batch", jobs=12, atoms_from=1000, atoms_to=12000, points_from=41,
             points_to=79, maps=6, mix=1),
        # Fitting the corrector: forward and backward over a training grid.
        dict(name="net_grad", path="net_grad", nx=81, ny=65, nz=57),
    ]


def _logint(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    path = rng.choice(["job", "job", "resident", "resident", "emap", "noalloc", "batch", "net_grad"])
    if path == "job":
        return dict(path="job", atoms=_logint(rng, 300, 20000), points=2 * _logint(rng, 12, 75) + 1,
                    maps=rng.choice([2, 6, 6, 10, 14]), diel=rng.choice([-0.1465, -0.1465, -0.1465, 40.0]),
                    spacing=rng.choice([0.375, 0.375, 0.25, 0.5]))
    if path == "resident":
        work = rng.choice(["all", "affinity", "emap", "surrogate"])
        atoms, most = (60000, 255) if work == "emap" else (20000, 161)
        return dict(path="resident", work=work, atoms=_logint(rng, 800, atoms),
                    nx=_logint(rng, 24, most), ny=_logint(rng, 24, most), nz=_logint(rng, 24, most),
                    maps=rng.choice([6, 10, 14]) if work in ("all", "affinity") else 0)
    if path == "emap":
        return dict(path="emap", atoms=_logint(rng, 300, 20000), nx=_logint(rng, 20, 150), ny=_logint(rng, 20, 150),
                    nz=_logint(rng, 20, 150))
    if path == "noalloc":
        return dict(path="noalloc", atoms=_logint(rng, 300, 20000), nx=_logint(rng, 20, 150),
                    ny=_logint(rng, 20, 150), nz=_logint(rng, 20, 150), diel=rng.choice([-0.1465, -0.1465, 40.0]))
    if path == "batch":
        return dict(path="batch", jobs=rng.randint(3, 14), atoms_from=1000, atoms_to=_logint(rng, 2000, 15000),
                    points_from=41, points_to=2 * _logint(rng, 22, 40) + 1, maps=rng.choice([2, 6]),
                    mix=rng.randint(1, 1000))
    return dict(path="net_grad", nx=_logint(rng, 24, 97), ny=_logint(rng, 24, 97), nz=_logint(rng, 24, 97))


# --- inputs ------------------------------------------------------------------------------------
def _problem(atoms, points, maps, diel, spacing, seed):
    """A parsed job on a seeded receptor (its files are read once and not needed again)."""
    r = 20.0 * (atoms / 2000.0) ** (1 / 3)
    axes = (1.2 * r, r, 0.85 * r) if atoms >= 5000 else (r, r, r)
    old = os.getcwd()
    with tempfile.TemporaryDirectory() as d:
        fg.synth_write(d, "rec", atoms, axes, points - 1, TYPES[maps], seed=seed, spacing=spacing, dielectric=diel)
        os.chdir(d)
        try:
            return fg.Problem("rec.gpf", log="rec.glg")
        finally:
            os.chdir(old)


def _job(case, seed):
    return _problem(case["atoms"], case["points"], case["maps"], case["diel"], case.get("spacing", 0.375), seed)


def _receptor(case, seed):
    """The job whose receptor a `resident` case computes on a grid of its own."""
    return _problem(case["atoms"], 31, case["maps"] or 2, -0.1465, 0.375, seed)


def _batch_sizes(case):
    """(atoms, points per axis) of each job: spread over both ranges, in an order of the case's own."""
    rng = np.random.default_rng(case["mix"])
    at = (np.arange(case["jobs"]) / (case["jobs"] - 1))
    atoms = np.rint(case["atoms_from"] * (case["atoms_to"] / case["atoms_from"]) ** at).astype(int)
    points = 2 * np.rint((case["points_from"] + (case["points_to"] - case["points_from"]) * at) / 2 - 0.5).astype(int) + 1
    return list(zip(rng.permutation(atoms).tolist(), rng.permutation(points).tolist()))


def _batch_jobs(case, seed):
    return [_problem(n, p, case["maps"], -0.1465, 0.375, 1000 * seed + i)
            for i, (n, p) in enumerate(_batch_sizes(case))]


def _atoms(case, seed, coeff=0.1465):
    return fg.surrogate_receptor(seed, case["atoms"]) * np.array([1.0, 1.0, 1.0, coeff / 0.1465])


def _net(case, seed):
    """Features (values that BF16 holds), a target, and weights of the size training starts from."""
    rng = np.random.default_rng([seed, 11])
    n = case["nx"] * case["ny"] * case["nz"]
    feat = torch.from_numpy(rng.standard_normal((n, 8)).astype(np.float32)).bfloat16().float().numpy()
    fan = [27 * 8, 27 * 32, 27 * 32]
    w = [rng.standard_normal(s).astype(np.float32) * np.float32(np.sqrt(2.0 / f))
         for s, f in zip((27 * 8 * 32, 27 * 32 * 32, 27 * 32), fan)]
    w = torch.from_numpy(np.concatenate(w)).bfloat16().float().numpy()
    target = rng.standard_normal(n).astype(np.float32)
    return feat, target, w


class _OnDevice:
    """A context's map set for torch (no copy; the context lives as long as the tensor)."""

    def __init__(self, ctx, n_sets, grid):
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=(n_sets, grid.nz, grid.ny, grid.nx), typestr="<f4",
                                             data=(ctx.device_maps(), False), version=3, strides=None)


class _OnHost:
    """A job's map set where ag_problem_compute leaves it, as the engine's own writers read it
    (no copy; the job lives as long as the array)."""

    def __init__(self, p):
        self.p = p
        at = ctypes.cast(fg.lib().ag_problem_maps(p.h), ctypes.c_void_p).value
        self.__array_interface__ = dict(shape=(p.n_maps + 2, p.grid.nz, p.grid.ny, p.grid.nx), typestr="<f4",
                                        data=(at, True), version=3)


WORK = dict(all=fg.AG_WORK_ALL, affinity=fg.AG_WORK_AFFINITY, emap=fg.AG_WORK_EMAP,
            surrogate=fg.AG_WORK_EMAP_SURROGATE)


def prepare(case, seed):
    path = case["path"]
    if path == "job":
        return dict(path=path, ctx=fg.Context(0), job=_job(case, seed))
    if path == "resident":
        ctx, p = fg.Context(0), _receptor(case, seed)
        grid = fg.Grid(case["nx"], case["ny"], case["nz"], 0.375)
        ctx.upload(grid, p.receptor, p.params if case["maps"] else None, p.inv_eps_ptr)
        if case["work"] == "surrogate":
            ctx.surrogate_load()
        maps = torch.as_tensor(_OnDevice(ctx, case["maps"] + 2, grid), device="cuda")
        return dict(path=path, ctx=ctx, job=p, work=case["work"], n=case["maps"], maps=maps)
    if path == "emap":
        grid = fg.Grid(case["nx"], case["ny"], case["nz"], 0.375)
        return dict(path=path, ctx=fg.Context(0), grid=grid, atoms=_atoms(case, seed), eps=fg.ddd_table())
    if path == "noalloc":
        grid = fg.Grid(case["nx"], case["ny"], case["nz"], 0.375)
        ddd = case["diel"] < 0
        atoms = _atoms(case, seed) if ddd else _atoms(case, seed, 332.0 / case["diel"])
        return dict(path=path, grid=grid, n=case["atoms"], atoms=torch.from_numpy(atoms).cuda(),
                    eps=torch.from_numpy(fg.ddd_table()).float().cuda() if ddd else None,
                    out=torch.empty(grid.nz, grid.ny, grid.nx, device="cuda"))
    if path == "batch":
        ctx, jobs = fg.Context(0), _batch_jobs(case, seed)
        return dict(path=path, ctx=ctx, batch=fg.Batch(ctx, jobs), jobs=len(jobs))
    ctx = fg.Context(0)
    feat, target, w = _net(case, seed)
    ctx.surrogate_weights(w, np.array([1.0, 1.0]))
    return dict(path=path, ctx=ctx, grid=fg.Grid(case["nx"], case["ny"], case["nz"], 0.375), feat=feat, target=target)


def run(state):
    path = state["path"]
    if path == "job":
        p = state["job"]
        p.compute(state["ctx"])
        maps = np.asarray(_OnHost(p))
        return dict(maps=maps[:p.n_maps], e=maps[p.n_maps], d=maps[p.n_maps + 1])
    if path == "resident":
        state["ctx"].compute(WORK[state["work"]])
        m, n = state["maps"], state["n"]
        if state["work"] == "all":
            return dict(maps=m[:n], e=m[n], d=m[n + 1])
        return dict(maps=m[:n], d=m[n + 1]) if state["work"] == "affinity" else dict(e=m[n])
    if path == "emap":
        return dict(e=state["ctx"].emap(state["grid"], state["atoms"], state["eps"]))
    if path == "noalloc":
        eps = state["eps"]
        rc = fg.lib().ag_emap_noalloc(ctypes.byref(state["grid"]), state["n"], state["atoms"].data_ptr(),
                                      None if eps is None else eps.data_ptr(), state["out"].data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)
        if rc != fg.AG_OK:
            raise fg.AgError(fg.lib().ag_last_error().decode(), rc)
        return dict(e=state["out"])
    if path == "batch":
        state["batch"].compute()
        return [state["batch"].maps(i) for i in range(state["jobs"])]
    o, grad, loss = state["ctx"].surrogate_net_grad(state["grid"], state["feat"], state["target"])
    return dict(o=o, grad=grad, loss=loss)


# --- what a pass cannot do without -------------------------------------------------------------
def _set_work(atoms, points, volume, maps, emap=True, affinity=True):
    """Inputs once and maps once; 12 operations per point-atom term of the defining e-map sum, and
    10 + 2 (maps + 1) per pair within 8 A (at the receptor's density of 0.06 atoms per A^3)."""
    out = (1 if emap else 0) + (maps + 1 if affinity else 0)
    w = dict(bytes=32.0 * atoms + 4.0 * out * points, flops=0.0)
    if emap:
        w["bytes"] += 4 * 8192
        w["flops"] += 12.0 * atoms * points
    if affinity:
        w["bytes"] += 72.0 * atoms + 4 * 801 * 6 * (maps + 1)
        inside = min(1.0, atoms / 0.06 / volume)  # share of the box that the receptor fills
        w["flops"] += 0.06 * 2144.7 * inside * points * (10 + 2 * (maps + 1))
    return w


def work(case):
    path = case["path"]
    if path == "job":
        n = case["points"] ** 3
        return _set_work(case["atoms"], n, n * case.get("spacing", 0.375) ** 3, case["maps"])
    if path == "batch":
        parts = [_set_work(a, p ** 3, p ** 3 * 0.375 ** 3, case["maps"]) for a, p in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    net = 2.0 * 27 * (8 * 32 + 32 * 32 + 32) * n
    if path == "net_grad":  # features, target, output; a forward pass and two products per layer behind it
        return dict(bytes=4.0 * n * 10 + 8.0 * 35424, flops=3 * net - 2.0 * 27 * 8 * 32 * n)
    if path == "resident" and case["work"] == "surrogate":
        near = 12.0 * 0.06 * 4188.8 * n        # the exact sum within 10 A
        far = 20.0 * case["atoms"] * n / 64    # the smooth sum on the 1.5 A grid
        return dict(bytes=32.0 * case["atoms"] + 4.0 * n + 4 * 8192, flops=near + far + net)
    what = case.get("work", "emap")
    return _set_work(case["atoms"], n, n * 0.375 ** 3, case.get("maps", 0), what != "affinity", what in ("all", "affinity"))


# --- the values in 64 bits ---------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _axes(nx, ny, nz, h):
    f = lambda n: (torch.arange(n, device=_dev(), dtype=torch.float64) - n // 2) * h  # noqa: E731
    return f(nx), f(ny), f(nz)


def _emap64(shape, h, xyzw, eps):
    """e(p) = sum w min(1/r, 2) eps[min(int(100 r), 8191)] over all atoms."""
    nx, ny, nz = shape
    a = torch.as_tensor(np.asarray(xyzw, dtype=np.float64), device=_dev())
    table = None if eps is None else torch.as_tensor(np.asarray(eps, dtype=np.float64), device=_dev())
    gx, gy, gz = _axes(nx, ny, nz, h)
    dx2 = (a[:, 0][None, :] - gx[:, None]) ** 2
    out = torch.empty(nz, ny, nx, dtype=torch.float64, device=_dev())
    rows = max(1, int(4e7 / (len(a) * nx)))
    for k in range(nz):
        dz2 = (a[:, 2] - gz[k]) ** 2
        for j in range(0, ny, rows):
            dyz = (a[:, 1][None, :] - gy[j:j + rows, None]) ** 2 + dz2
            r = (dx2[None] + dyz[:, None]).sqrt_()
            t = (1.0 / r).clamp_(max=2.0)
            if table is not None:
                t *= table[(r * 100.0).long().clamp_(max=8191)]
            out[k, j:j + rows] = t @ a[:, 3]
    return out


def _views(p):
    """The loader's arrays as tensors."""
    n, nm, nt = p.info.n_atoms, p.n_maps, p.params.n_types
    r, q = p.receptor, p.params

    def get(ptr, *shape):
        v = np.ctypeslib.as_array(ptr, shape=shape).copy()
        return torch.as_tensor(v.astype(np.float64 if v.dtype.kind == "f" else np.int64), device=_dev())

    return dict(xyz=get(r.xyzw, n, 4)[:, :3].contiguous(), q=get(r.charge, n), vol=get(r.vol, n),
                solpar=get(r.solpar, n), type=get(r.type, n), hb=get(r.hbond, n), dis=get(r.disorder, n) != 0,
                rexp=get(r.rexp, n), rv=get(r.rvector, n, 3), rv2=get(r.rvector2, n, 3),
                energy=get(q.energy, nt, 8192, nm), sol=get(q.sol, 8192), mhb=get(q.map_hbond, nm).tolist(),
                mis=get(q.map_is_hbonder, nm).tolist(), psol=get(q.solpar_probe, nm), pvol=get(q.vol_probe, nm),
                sq=q.solpar_q, hydrogen=q.hydrogen)


DS, D1, AS, A1, A2 = 1, 2, 3, 4, 5  # AutoGrid's H-bond classes


def _angular64(v, atom, donor, u):
    """The directional factors (racc, rdon, Hramp) of each pair."""
    pi = np.pi
    one = torch.ones_like(u[:, 0])
    racc, rdon, ramp = one.clone(), one.clone(), one.clone()
    rv, rv2, hb, dis = v["rv"][atom], v["rv2"][atom], v["hb"][atom], v["dis"][atom]
    cos = -(u * rv).sum(1)
    acos = lambda x: x.clamp(-1, 1).acos()  # noqa: E731
    c2 = cos * cos
    power = torch.where(v["rexp"][atom] == 4, c2 * c2, torch.where(v["rexp"][atom] == 2, c2, cos))
    d1 = hb == D1
    racc = torch.where(d1, torch.where(cos > 0, power, 0 * one), racc)
    turn = 0.5 - 0.5 * torch.cos(acos((v["rv"][donor] * rv).sum(1)) * (120.0 / 90.0))
    ramp = torch.where(d1 & (cos > 0) & (atom != donor), turn, ramp)
    rdon = torch.where(hb == A1, torch.where(cos > 0, c2, 0 * one), rdon)
    a2 = hb == A2
    theta = acos(cos)
    loose = torch.where(theta <= 1.24791 + pi / 2, torch.cos(theta - 1.24791) ** 4, 0 * one)
    cr = torch.linalg.cross(u, rv2)
    ti = (acos((cr * rv).sum(1) / (cr * cr).sum(1).clamp(min=1e-6).sqrt()) - pi / 2).abs()
    rd = torch.where(cos >= 0, 0.9 + 0.1 * torch.sin(2 * ti),
                     torch.where(cos >= -0.34202, 562.25 * (0.116978 - c2) ** 3, 0 * one))
    tight = rd * torch.cos(pi / 2 - acos((u * rv2).sum(1)))
    rdon = torch.where(a2, torch.where(dis, loose, tight), rdon)
    racc = torch.where(a2 & dis, loose, racc)
    return racc, rdon, ramp


def _affinity64(shape, h, v):
    """The affinity maps and the desolvation map: pairs within 8 A, tables in 0.01 A bins, the
    directional H-bond terms (sums for acceptor probes at donors, minimum plus maximum else)."""
    nx, ny, nz = shape
    gx, gy, gz = _axes(nx, ny, nz, h)
    nm, dev = v["energy"].shape[2], _dev()
    maps = torch.zeros(nm, nz, ny * nx, dtype=torch.float64, device=dev)
    dmap = torch.zeros(nz, ny * nx, dtype=torch.float64, device=dev)
    donors = torch.nonzero((v["hb"] == DS) | (v["hb"] == D1))[:, 0]
    py, px = gy.repeat_interleave(nx), gx.repeat(ny)
    for k in range(nz):
        near = torch.nonzero((v["xyz"][:, 2] - gz[k]).abs() <= 8.0)[:, 0]
        dons = donors[(v["xyz"][donors, 2] - gz[k]).abs() <= 8.0]
        if len(near) == 0:
            continue
        step = max(1, int(3e7 / len(near)))
        for s in range(0, nx * ny, step):
            qx, qy = px[s:s + step], py[s:s + step]
            m = len(qx)

            def rsq(i):
                x = v["xyz"][i]
                return ((x[:, 0][None] - qx[:, None]) ** 2 + (x[:, 1][None] - qy[:, None]) ** 2) + \
                    (x[:, 2] - gz[k])[None] ** 2

            best = torch.zeros(m, dtype=torch.int64, device=dev)
            if len(dons):
                r2 = rsq(dons)
                low = r2.amin(1, keepdim=True)
                best = torch.where(r2 == low, dons[None], len(v["q"])).amin(1)  # ties: the first in the file
            r2 = rsq(near)
            keep = r2 <= 64.0
            keep &= ~((v["type"][near] == v["hydrogen"]) & v["dis"][near])[None]
            pt, ia = torch.nonzero(keep, as_tuple=True)
            if len(pt) == 0:
                continue
            r2 = r2[pt, ia].clamp(min=1e-24)
            atom = near[ia]
            inv = 1.0 / r2.sqrt()
            d = v["xyz"][atom] - torch.stack([qx[pt], qy[pt], gz[k].expand(len(pt))], 1)
            b = ((1.0 / inv) * 100.0).long().clamp(max=8191)
            racc, rdon, ramp = _angular64(v, atom, best[pt], d * inv[:, None])
            hb, t = v["hb"][atom], v["type"][atom]
            isdon, isacc = (hb == DS) | (hb == D1), hb >= AS
            sol = v["sol"][b]
            s1, s2 = v["vol"][atom] * sol, (v["solpar"][atom] + v["sq"] * v["q"][atom].abs()) * sol
            dmap[k].index_add_(0, pt + s, v["sq"] * s1)
            for g in range(nm):
                e = v["energy"][t, b, g]
                acc = v["psol"][g] * s1 + v["pvol"][g] * s2
                sph = (e / 100).clamp(0, 1)
                mhb = v["mhb"][g] if v["mis"][g] else 0
                if mhb in (AS, A2):
                    far = v["energy"][max(v["hydrogen"], 0), (b - 110).clamp(min=0), g]
                    bond = torch.where(v["dis"][atom], far, e) * ramp * (racc + (1 - racc) * sph)
                    acc = acc + torch.where(isdon, bond, e)
                elif mhb in (DS, D1, A1):
                    here, f = (isdon, racc) if mhb == A1 else (isacc, rdon)
                    val = (e * (f + (1 - f) * sph))[here]
                    acc = acc + torch.where(here, 0 * e, e)
                    lo = torch.full((m,), 999999.0, dtype=torch.float64, device=dev)
                    hi = -lo
                    lo.scatter_reduce_(0, pt[here], val, "amin")
                    hi.scatter_reduce_(0, pt[here], val, "amax")
                    maps[g, k, s:s + m] += torch.where(lo < 999999.0, lo + hi, 0 * lo)
                else:
                    acc = acc + e
                maps[g, k].index_add_(0, pt + s, acc)
    return maps.view(nm, nz, ny, nx), dmap.view(nz, ny, nx)


def _net64(case, seed):
    feat, target, w = (torch.from_numpy(a).to(_dev(), torch.float64) for a in _net(case, seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    w = w.requires_grad_()
    w1, w2, w3 = w.split([27 * 8 * 32, 27 * 32 * 32, 27 * 32])
    x = feat.view(nz, ny, nx, 8)

    def conv(x, k, cin, cout):  # a 3x3x3 window as 27 products, zero outside the grid
        p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        k = k.view(27, cin, cout)
        return sum(p[t // 9:t // 9 + nz, t // 3 % 3:t // 3 % 3 + ny, t % 3:t % 3 + nx] @ k[t] for t in range(27))

    act = lambda z: torch.where(z > 0, z, z / 8)  # noqa: E731
    o = conv(act(conv(act(conv(x, w1, 8, 32)), w2, 32, 32)), w3, 32, 1).reshape(-1)
    loss = ((o - target) ** 2).mean()
    loss.backward()
    return dict(o=o.detach(), grad=w.grad, loss=float(loss.detach()))


def exact(case, seed):
    path = case["path"]
    if path == "net_grad":
        return _net64(case, seed)
    if path == "batch":
        out = []
        for p in _batch_jobs(case, seed):
            shape = (p.grid.nx, p.grid.ny, p.grid.nz)
            maps, d = _affinity64(shape, p.grid.spacing, _views(p))
            e = _emap64(shape, p.grid.spacing, p.xyzw(), p.inv_eps())
            out.append(torch.cat([maps, e[None], d[None]]))
        return out
    if path == "job":
        p, n = _job(case, seed), case["points"]
        shape, h = (n, n, n), p.grid.spacing
        if n ** 3 * case["atoms"] > 1.5e11:
            return None
        maps, d = _affinity64(shape, h, _views(p))
        return dict(maps=maps, e=_emap64(shape, h, p.xyzw(), p.inv_eps()), d=d)
    shape = (case["nx"], case["ny"], case["nz"])
    if shape[0] * shape[1] * shape[2] * case["atoms"] > 1.5e11:
        return None
    if path == "resident":
        p = _receptor(case, seed)
        out = {}
        if case["work"] in ("all", "affinity"):
            out["maps"], out["d"] = _affinity64(shape, 0.375, _views(p))
        if case["work"] != "affinity":
            out["e"] = _emap64(shape, 0.375, p.xyzw(), p.inv_eps())
        return out
    ddd = path == "emap" or case["diel"] < 0
    atoms = _atoms(case, seed) if ddd else _atoms(case, seed, 332.0 / case["diel"])
    e = _emap64(shape, 0.375, atoms, fg.ddd_table() if ddd else None)
    return dict(e=e.view(-1) if path == "emap" else e)
