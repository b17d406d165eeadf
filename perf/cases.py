"""What the speed of the library is measured on: its public entry points over the range they are used in.

A case is a dict of plain values; `kind` says which entry point it goes through:

- "level": one substep of a uniform periodic 3D level (`Context.level_substep`, a captured graph) -- the time loop of
  a uniform run, state resident on the device, the step from the CFL reduction;
- "host": the same substep on state in page-locked host memory (`Context.level_substep_host_ptr`) -- an application
  that keeps its arrays on the host;
- "run1d": a whole 1D Sod-like run from its upload to its end time (`Context.level_run`);
- "boxes": one substep of an ensemble of uneven independent boxes, a CFL step per box;
- "amr": a run resumed from a saved tree and state (`Context.tree_attach`), several coarse steps with sub-cycling,
  refinement and removal on the device (`DeviceAmrRun.coarse_step`), the state read back at the end;
- "exact": a batch of exact Riemann solves (`Context.exact_batch`), as the reference stops Newton or converged, from
  the two-shock or the learned start;
- "grad": loss gradients of the start network (`Context.mlp_grad`), its training kernel's forward and backward pass.

Sizes: edges of the level cases are nx 2^(level-1) cells.  Every state is made on the GPU from the seed.
"""
import functools
import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "ramses-cpp_b200"))

import rg_amr  # noqa: E402
import rg_ensemble  # noqa: E402
import rg_tree  # noqa: E402
import rgpu  # noqa: E402

F8 = torch.float64


def listed():
    lv = dict(kind="level", slope=2, riemann="hllc", interp=1)
    return [
        # the smallest 3D step: launches and the graph count, not the cells
        dict(lv, name="level_16", nx=1, level=5),
        # a ragged base grid (nx = 3, dx no power of two), the default slopes and solver of the namelist
        dict(lv, name="level_48_llf", nx=3, level=5, slope=1, riemann="llf"),
        # the ordinary uniform run: the AMR run's base grid
        dict(lv, name="level_64", nx=1, level=7),
        # the uniform Sedov configuration's grid
        dict(lv, name="level_128", nx=1, level=8),
        # the exact solver on a base grid that is no power of two
        dict(lv, name="level_96_exact", nx=3, level=6, riemann="exact"),
        # an application with its state on the host: the copies over the bus count too
        dict(lv, name="host_64", kind="host", nx=1, level=7),
        # the Sod configuration, from upload to t = 0.245
        dict(name="run1d_1024", kind="run1d", level=11, slope=1, riemann="hllc", interp=1, tend=0.245),
        # uneven boxes stepped together, the ensemble configuration in small
        dict(name="boxes_40", kind="boxes", nbox=40, pick=20261203, slope=2, riemann="hllc", interp=1),
        # the Sedov AMR configuration (64^3 base, 512^3 effective), a window of its coarse steps after a restart
        dict(name="amr_7_10", kind="amr", lmin=7, lmax=10, steps=20),
        # a small AMR run, where waits and launches count
        dict(name="amr_5_7", kind="amr", lmin=5, lmax=7, steps=8),
        # exact solves as the reference stops them, and converged from the learned start (the stress workload)
        dict(name="exact_4m", kind="exact", n=1 << 22, mode="reference", learned=False),
        dict(name="exact_4m_learned", kind="exact", n=1 << 22, mode="converged", learned=True),
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    kind = rng.choice(["level", "level", "level", "host", "run1d", "boxes", "amr", "exact", "exact", "grad"])
    phys = dict(slope=rng.choice([1, 2, 2, 8]), riemann=rng.choice(["hllc", "hllc", "hll", "llf", "exact"]), interp=1)
    if kind in ("level", "host"):
        top = 128 if kind == "level" else 64
        shapes = [(nx, lev) for nx in (1, 3, 5, 7) for lev in range(3, 9) if 8 <= nx << (lev - 1) <= top]
        edge = math.exp(rng.uniform(math.log(8), math.log(top + 1)))
        nx, lev = min(shapes, key=lambda s: (abs(math.log((s[0] << (s[1] - 1)) / edge)), rng.random()))
        return dict(phys, kind=kind, nx=nx, level=lev, interp=rng.choice([1, 1, 2, 3]))
    if kind == "run1d":
        return dict(kind=kind, level=rng.choice([7, 8, 9, 10, 11, 12]), slope=rng.choice([1, 2]),
                    riemann=rng.choice(["hllc", "hll", "llf"]), interp=1, tend=round(rng.uniform(0.02, 0.1), 4))
    if kind == "boxes":
        return dict(kind=kind, nbox=int(math.exp(rng.uniform(math.log(2), math.log(40)))),
                    pick=rng.randrange(1 << 20), slope=rng.choice([1, 2]), riemann=rng.choice(["hllc", "hll"]),
                    interp=1)
    if kind == "amr":
        lmin = rng.choice([4, 5, 6])
        return dict(kind=kind, lmin=lmin, lmax=lmin + rng.choice([1, 2, 3]), steps=rng.randint(4, 12))
    n = int(math.exp(rng.uniform(math.log(100), math.log(1 << 22))))
    if kind == "exact":
        return dict(kind=kind, n=n, mode=rng.choice(["reference", "converged"]), learned=rng.random() < 0.4)
    return dict(kind=kind, n=min(n, 1 << 17))


# ---------------------------------------------------------------- layouts, kept between cases as a program keeps them

@functools.lru_cache(maxsize=8)
def _uniform(ndim, nx, level):
    """The tree of a uniform level, and per lattice site (x fastest) its cell's index and its place in the loop order."""
    n3 = nx if ndim == 3 else 1
    g = rg_tree.build_uniform(ndim, level, nx=nx, ny=n3, nz=n3)
    edge = nx << (level - 1)
    ids = g.cell_ids(level)
    ijk = np.rint(g.cell_centers(level) * edge - 0.5).astype(np.int64)
    site = ijk[:, 0] if ndim == 1 else ijk[:, 0] + edge * (ijk[:, 1] + edge * ijk[:, 2])
    cell = np.zeros(len(ids), np.int64)
    order = np.zeros(len(ids), np.int64)
    cell[site] = ids - 1
    order[site] = np.arange(len(ids))
    above = np.concatenate([g.cell_ids(lev) for lev in range(2, level)]) - 1 if level > 2 else np.zeros(0, np.int64)
    return SimpleNamespace(g=g, edge=edge, dx=1.0 / (nx * 2.0 ** level), cell=torch.from_numpy(cell).cuda(),
                           order=torch.from_numpy(order).cuda(), above=torch.from_numpy(above).cuda())


@functools.lru_cache(maxsize=3)
def _forest(nbox, pick):
    specs = rg_ensemble.box_specs(nbox, seed=pick)
    f = rg_ensemble.Forest(specs)
    ext, lat_id, lat_p = f.lattices()
    noct = int(f.first_oct[-1])
    k, ic = lat_p % noct, lat_p // noct
    return SimpleNamespace(f=f, ext=ext, lat_id=lat_id, lat_p=lat_p, cell=torch.from_numpy(lat_id.astype(np.int64) - 1).cuda(),
                           order=torch.from_numpy(k.astype(np.int64) * 8 + ic).cuda())


def _rand(seed, n):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    return torch.rand(n, generator=gen, device="cuda", dtype=F8)


class _Raw:
    """A device array of the library as something torch can take a view of; the view keeps the context alive."""

    def __init__(self, ctx, ptr, n):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _views(ctx, n):
    a, b = ctx.device_state()
    return torch.as_tensor(_Raw(ctx, a, n), device="cuda"), torch.as_tensor(_Raw(ctx, b, n), device="cuda")


def _cons(rho, vel, p, gamma):
    """Conservative variables [nvar][n] of primitive ones."""
    return torch.stack([rho] + [rho * v for v in vel] + [p / (gamma - 1.0) + 0.5 * rho * sum(v * v for v in vel)])


def _params(case, ndim, gamma):
    return rgpu.make_params(ndim, slope_type=case["slope"], riemann=case["riemann"], interpol_type=case["interp"],
                            gamma=gamma, courant_factor=0.8)


# ---------------------------------------------------------------- inputs

def _flow3d(lay, seed):
    """A blast in a gas with waves: a few random Fourier modes of density and velocity, and a ball of high pressure."""
    e = lay.edge
    x = (torch.arange(e, device="cuda", dtype=F8) + 0.5) / e
    r = _rand(seed, 64).tolist()

    def modes(o):
        w = 0.0
        for m in range(3):
            a = 2 * math.pi * (r[o + 4 * m] + (1 + m % 2) * x)[None, None, :]
            b = 2 * math.pi * (r[o + 4 * m + 1] + (1 + (m + 1) % 2) * x)[None, :, None]
            c = 2 * math.pi * (r[o + 4 * m + 2] + x)[:, None, None]
            w = w + (r[o + 4 * m + 3] - 0.5) * torch.sin(a) * torch.sin(b) * torch.sin(c)
        return w
    c = [0.4 + 0.2 * v for v in r[60:63]]
    d2 = (x[None, None, :] - c[0]) ** 2 + (x[None, :, None] - c[1]) ** 2 + (x[:, None, None] - c[2]) ** 2
    rho = torch.exp(0.8 * modes(0))
    p = torch.where(d2 < (0.1 + 0.5 / e) ** 2, 20.0, 0.5) * torch.exp(0.5 * modes(12))
    vel = [0.8 * modes(24 + 12 * k) for k in range(3)]
    return _cons(rho.reshape(-1), [v.reshape(-1) for v in vel], p.reshape(-1), 1.4)


def _flow1d(lay, seed):
    """Sod's tube with the states and the place of the jump moved a little by the seed."""
    r = _rand(seed, 4).tolist()
    x = (torch.arange(lay.edge, device="cuda", dtype=F8) + 0.5) / lay.edge
    left = x < 0.45 + 0.1 * r[0]
    rho = torch.where(left, 0.9 + 0.2 * r[1], 0.125)
    p = torch.where(left, 0.9 + 0.2 * r[2], 0.1 + 0.02 * r[3])
    return _cons(rho, [torch.zeros_like(x)], p, 1.4)


def _flow_boxes(fo, seed):
    """The ensemble's planar Riemann problems: random normals and states, one per box, in lattice order."""
    r = _rand(seed, 16 * fo.f.nbox).reshape(-1, 16).tolist()
    parts = []
    for s, q in zip(fo.f.specs, r):
        x = (torch.arange(s.edge, device="cuda", dtype=F8) + 0.5) / s.edge - 0.5
        th, ph = math.acos(2 * q[0] - 1), 2 * math.pi * q[1]
        nrm = (math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th))
        left = (nrm[0] * x[None, None, :] + nrm[1] * x[None, :, None] + nrm[2] * x[:, None, None]).reshape(-1) < 0
        side = [(10 ** (6 * q[o] - 3), 6 * q[o + 1] - 3, 10 ** (8 * q[o + 2] - 4)) for o in (2, 5)]
        rho, un, p = (torch.where(left, a, b) for a, b in zip(*side))
        parts.append(_cons(rho.to(F8), [un * c for c in nrm], p.to(F8), 5.0 / 3.0))
    return torch.cat(parts, dim=1)


def _level_full(lay, u):
    """The library's [nvar][ncell] state with `u` on the level's cells, and unit gas at rest on the cells above."""
    g, nv = lay.g, u.shape[0]
    full = torch.zeros(nv, g.ncell, device="cuda", dtype=F8)
    full[0, lay.above] = 1.0
    full[nv - 1, lay.above] = 2.5
    full[:, lay.cell] = u
    return full.reshape(-1)


def _fill(views, full):
    for v in views:
        v.copy_(full)
    torch.cuda.synchronize()


def _prepare_level(case, seed, ndim):
    lay = _uniform(ndim, case.get("nx", 1), case["level"])
    full = _level_full(lay, _flow3d(lay, seed) if ndim == 3 else _flow1d(lay, seed))
    ctx = rgpu.Context(_params(case, ndim, 1.4), 0)
    ctx.sync_topology(lay.g)
    views = _views(ctx, full.numel())
    _fill(views, full)
    L, dx = case["level"], lay.dx
    for _ in range(2):  # the plan, the face kernel's shape and the graph, which a program keeps for its run
        ctx.level_substep(L, dx)
    ctx.synchronize()
    if case["kind"] == "host":
        host = torch.empty(full.numel(), dtype=F8, pin_memory=True)
        host.copy_(full)
        ctx.level_substep_host_ptr(L, dx, host.data_ptr(), want_dt=False)
        host.copy_(full)
        return dict(kind="host", ctx=ctx, L=L, dx=dx, host=host)
    views = _views(ctx, full.numel())  # the state is set anew: the next substep starts from it
    _fill(views, full)
    if ndim == 1:
        u0 = full.cpu().numpy()
        return dict(kind="run1d", ctx=ctx, L=L, dx=dx, uold=views[0], u0=u0, tend=case["tend"])
    return dict(kind="level", ctx=ctx, L=L, dx=dx, uold=views[0])


def _prepare_boxes(case, seed):
    fo = _forest(case["nbox"], case["pick"])
    f = fo.f
    full = torch.zeros(5, f.grid.ncell, device="cuda", dtype=F8)
    full[:, fo.cell] = _flow_boxes(fo, seed)
    full = full.reshape(-1)
    ctx = rgpu.Context(_params(case, 3, 5.0 / 3.0), 0)
    ctx.sync_topology(f.grid)
    views = _views(ctx, full.numel())
    _fill(views, full)
    ctx.set_level_boxes(f.level, f.first_oct, f.dx)
    ctx.set_level_lattices(f.level, fo.ext, fo.lat_id, fo.lat_p)
    for _ in range(2):
        ctx.level_substep(f.level, 0.0)
    ctx.synchronize()
    views = _views(ctx, full.numel())
    _fill(views, full)
    return dict(kind="level", ctx=ctx, L=f.level, dx=0.0, uold=views[0])


AMR_CFL, AMR_ERR = 0.25, 0.1


def _prepare_amr(case, seed):
    """The Sedov run's tree and state after its initialisation, in host arrays as a restart file gives them."""
    r = _rand(seed, 3).tolist()
    lmin, lmax = case["lmin"], case["lmax"]
    ngridmax = sum(8 ** (lev - 2) for lev in range(2, lmin + 1)) + 10551
    ctx = rgpu.Context(rgpu.make_params(3, slope_type=2, riemann="hllc", gamma=1.4, courant_factor=AMR_CFL), 0)
    ic = rg_amr.sedov_primitives(3, lmin, 1.4, rho0=0.9 + 0.2 * r[0], p0=1e-5 * (0.5 + r[1]), e_blast=0.9 + 0.2 * r[2])
    rg_amr.initialize(ctx, 3, lmin, lmax, ngridmax, ic, 1.4, ed=AMR_ERR, ep=AMR_ERR)
    like = rg_tree.tree_arrays(rg_tree.build_uniform(3, lmin, ngridmax=ngridmax, nlevelmax=lmax))
    arrays = ctx.tree_fetch({k: like[k] for k in ("headl", "taill", "numbl")})
    ngm, ncell = ctx.tree_sizes()
    g = rg_tree.Grid(ndim=3, nx=1, ny=1, nz=1, ngridmax=ngm, nlevelmax=lmax, nvar=5, levelmin=lmin)
    g.son, g.father, g.nbor, g.next, g.headl, g.xg = (arrays[k] for k in ("son", "father", "nbor", "next", "headl", "xg"))
    return dict(kind="amr", ctx=ctx, g=g, arrays=arrays, case=dict(case), out=np.empty(5 * ncell), ncell=ncell)


@functools.lru_cache(maxsize=1)
def _network():
    ctx = rgpu.Context(rgpu.make_params(3, riemann="exact"), 0)
    ctx.mlp_train(nsamples=1_000_000, epochs=10)
    w = ctx.mlp_get()
    ctx.close()
    return w


def _stress(n, seed):
    """Interface pairs of the stress workload: density ratios to 1e4, pressure ratios to 1e6, 30 % strong rarefactions."""
    r = _rand(seed, 16 * n).reshape(16, n)
    gam = torch.where(r[0] < 0.5, 5.0 / 3.0, 1.4).to(F8)
    rl = 10 ** (4 * r[1] - 2)
    rr = (rl * 10 ** (8 * r[2] - 4)).clamp(1e-4, 1e4)
    pl = 10 ** (6 * r[3] - 3)
    pr = (pl * 10 ** (12 * r[4] - 6)).clamp(1e-6, 1e6)
    du = (0.2 + 1.3 * r[6]) * 2 * ((gam * pl / rl).sqrt() + (gam * pr / rr).sqrt()) / (gam - 1)
    f = 0.2 + 0.6 * r[7]
    rare = r[5] < 0.3
    ul = torch.where(rare, -f * du, 6 * r[6] - 3)
    ur = torch.where(rare, (1 - f) * du, 6 * r[7] - 3)
    t = 2 * r[8:12] - 1
    return torch.stack([rl, ul, t[0], t[1], pl]), torch.stack([rr, ur, t[2], t[3], pr]), gam


def _prepare_exact(case, seed):
    n = case["n"]
    ctx = rgpu.Context(rgpu.make_params(3, riemann="exact"), 0)
    if case["learned"]:
        ctx.mlp_set(_network())
    ql, qr, gam = _stress(n, seed)
    st = dict(kind="exact", ctx=ctx, n=n, ql=ql, qr=qr, gam=gam, flux=torch.empty(5, n, device="cuda", dtype=F8),
              pstar=torch.empty(n, device="cuda", dtype=F8), iters=torch.empty(n, device="cuda", dtype=torch.int32))
    st["kw"] = dict(learned=case["learned"], niter=10 if case["mode"] == "reference" else 100,
                    tol=1e-6 if case["mode"] == "reference" else 1e-14)
    torch.cuda.synchronize()
    return st


def _prepare_grad(case, seed):
    n = case["n"]
    r = _rand(seed, 9 * n).reshape(9, n)
    x = (3.4 * (r[:8] - 0.5)).float().cpu().numpy()
    t = (3.4 * (r[8] - 0.5)).float().cpu().numpy()
    ctx = rgpu.Context(rgpu.make_params(3, riemann="exact"), 0)
    ctx.mlp_set(_network())
    return dict(kind="grad", ctx=ctx, x=x, t=t)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("level", "host"):
        return _prepare_level(case, seed, 3)
    if kind == "run1d":
        return _prepare_level(case, seed, 1)
    return {"boxes": _prepare_boxes, "amr": _prepare_amr, "exact": _prepare_exact, "grad": _prepare_grad}[kind](case, seed)


# ---------------------------------------------------------------- one pass

def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "level":
        ctx.level_substep(s["L"], s["dx"])
        return s["uold"]
    if kind == "host":
        ctx.level_substep_host_ptr(s["L"], s["dx"], s["host"].data_ptr(), want_dt=False)
        return s["host"]
    if kind == "run1d":
        ctx.upload_state(s["u0"], s["u0"])
        t, n = ctx.level_run(s["L"], s["dx"], s["tend"], pressure_cap=True)
        return [s["uold"], t, n]
    if kind == "amr":
        c = s["case"]
        ctx.tree_attach(s["g"], s["arrays"], c["lmin"])
        r = rg_amr.DeviceAmrRun(ctx, nx=1, levelmin=c["lmin"], nlevelmax=c["lmax"], cfl=AMR_CFL, ed=AMR_ERR, ep=AMR_ERR)
        for _ in range(c["steps"]):
            r.coarse_step()
        ncell = ctx.tree_sizes()[1]
        if s["out"].size != 5 * ncell:  # the tree grew
            s["out"] = np.empty(5 * ncell)
        ctx.download_state(uold=s["out"])
        return [s["out"], r.t, r.cell_updates] + [ctx.level_octs(L) for L in range(c["lmin"] + 1, c["lmax"] + 1)]
    if kind == "exact":
        ctx.exact_batch(s["n"], s["ql"].data_ptr(), s["qr"].data_ptr(), s["gam"].data_ptr(), s["flux"].data_ptr(),
                        s["pstar"].data_ptr(), s["iters"].data_ptr(), **s["kw"])
        return [s["flux"], s["pstar"], s["iters"]]
    g, loss = ctx.mlp_grad(s["x"], s["t"])
    return [g, loss]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Bytes: the state read once and written once (80 B per 3D cell update, 48 B in 1D), or the arrays of a batch.
    Operations: the scheme's own, a division or root counted once: about 1400 per 3D cell update with the cheap
    solvers, 250 per Newton solve."""
    kind = case["kind"]
    if kind in ("level", "host"):
        cells = (case["nx"] << (case["level"] - 1)) ** 3
        return {"bytes": 80 * cells, "flops": (1400 if case["riemann"] != "exact" else 2000) * cells}
    if kind == "run1d":
        n = 1 << (case["level"] - 1)
        updates = n * case["tend"] * 7.0 * n  # about 1729 substeps of 1024 cells to t = 0.245
        return {"bytes": 48 * n, "flops": 280 * updates}
    if kind == "boxes":
        cells = sum(s.cells for s in rg_ensemble.box_specs(case["nbox"], seed=case["pick"]))
        return {"bytes": 80 * cells, "flops": 1400 * cells}
    if kind == "amr":
        # base cells once, the finest level's (640 cells one level down, eight times as many per further level) at
        # each of its sub-steps
        nl = case["lmax"] - case["lmin"]
        base = 8 ** (case["lmin"] - 1)
        updates = case["steps"] * (base + 640 * 8 ** (nl - 1) * 2 ** nl)
        return {"bytes": 80 * updates + 120 * base, "flops": 1400 * updates}
    if kind == "exact":
        return {"bytes": (5 * 8 * 3 + 8 + 8 + 4) * case["n"], "flops": (250 if case["mode"] == "reference" else 400) * case["n"]}
    return {"bytes": 4 * 9 * case["n"], "flops": 6 * 4736 * case["n"]}


def tolerance(case):
    # One substep against plain torch is 2e-16 off, a batch of solves 6e-16 (converged, learned start), the BF16
    # gradients 3e-3.  The long runs are exact: the scheme grows rounding at a shock by a factor of 1e5 in 80
    # substeps (1D run against plain torch, substep by substep), so after a thousand of them nothing but the same
    # bits says that two runs are the same run; the library promises the reference's bits.
    return {"level": {"rel": 1e-15}, "host": {"rel": 1e-15}, "run1d": "exact", "boxes": {"rel": 1e-15},
            "amr": "exact", "exact": {"rel": 3e-15, "differ": 1e-5}, "grad": {"rel": 1.5e-2}}[case["kind"]]


# ---------------------------------------------------------------- the same in plain torch, 64 bits

def _prim(u, gamma):
    nd = u.shape[0] - 2
    d = u[0].clamp_min(1e-10)
    v = [u[1 + i] / d for i in range(nd)]
    eint = (u[nd + 1] / d - 0.5 * sum(a * a for a in v)).clamp_min(1e-20 / gamma / (gamma - 1))
    return torch.stack([d] + v + [(gamma - 1) * d * eint])


def _slope(l, c, r, kind):
    a, b = c - l, r - c
    if kind == 1:
        lim = torch.minimum(a.abs(), b.abs())
    else:
        th = 2.0 if kind == 2 else 1.5
        lim = torch.minimum(torch.minimum(th * a.abs(), th * b.abs()), (0.5 * (a + b)).abs())
    return torch.where(a * b > 0, torch.sign(a + b) * lim, torch.zeros_like(a))


def _interp(l, c, r, kind):
    a, b = c - l, r - c
    lim = {1: lambda: 0.5 * torch.minimum(a.abs(), b.abs()),
           2: lambda: torch.minimum(torch.minimum(a.abs(), b.abs()), 0.25 * (a + b).abs()),
           3: lambda: 0.25 * (a + b).abs()}[kind]()
    return torch.where(a * b > 0, torch.sign(a) * lim, torch.zeros_like(a))


def _trace(q, dq, dt, dx, gamma):
    """Half-step predicted states at a cell's lower and upper faces; normal velocity in slot 1."""
    ip = q.shape[0] - 1
    r = q[0].clamp_min(1e-10)
    p = torch.maximum(q[ip], r * 1e-20)
    src = torch.zeros_like(q)
    src[0] = -q[1] * dq[0] - dq[1] * r
    src[1] = -q[1] * dq[1] - dq[ip] / r
    src[ip] = -q[1] * dq[ip] - dq[1] * r * (gamma * p / r).clamp_min(1e-20)
    lo, hi = q - 0.5 * dx * dq + 0.5 * dt * src, q + 0.5 * dx * dq + 0.5 * dt * src
    for f in (lo, hi):
        f[0] = torch.where(f[0] < 1e-10, r, f[0])
    return lo, hi


def _energy(q, gamma):
    return q[-1] / (gamma - 1) + 0.5 * q[0] * (q[1:-1] ** 2).sum(0)


def _flux_of(q, gamma):
    m = q[0] * q[1]
    return torch.stack([m, m * q[1] + q[-1]] + [m * t for t in q[2:-1]] + [(_energy(q, gamma) + q[-1]) * q[1]])


def _cons_of(q, gamma):
    return torch.stack([q[0]] + [q[0] * v for v in q[1:-1]] + [_energy(q, gamma)])


def _sound(r, p, gamma):
    return (gamma * p / r).clamp_min(1e-20).sqrt()


def _riemann_exact(ql, qr, gamma, niter, tol, root=False):
    """The two-shock Newton solver; `root`: its converged root instead of the reference's stop."""
    sp = 1e-20 / gamma
    rl, rr, ul, ur = ql[0].clamp_min(1e-10), qr[0].clamp_min(1e-10), ql[1], qr[1]
    pl, pr = torch.maximum(ql[-1], rl * sp), torch.maximum(qr[-1], rr * sp)
    g6 = (gamma + 1) / (2 * gamma)
    cl, cr = gamma * pl * rl, gamma * pr * rr
    wl, wr = cl.sqrt(), cr.sqrt()

    def mass(p):
        return (cl * (1 + g6 * (p - pl) / (pl + 1e-20))).clamp_min(0).sqrt(), (cr * (1 + g6 * (p - pr) / (pr + 1e-20))).clamp_min(0).sqrt()

    def update(p):
        a, b = mass(p)
        x, y = 2 * a ** 3 / (a * a + cl + 1e-20), 2 * b ** 3 / (b * b + cr + 1e-20)
        gap = (ul - (p - pl) / (a + 1e-20)) - (ur + (p - pr) / (b + 1e-20))
        return torch.maximum(y * x / (y + x + 1e-20) * gap, -p), gap
    p = ((wr * pl + wl * pr + wl * wr * (ul - ur)) / (wl + wr + 1e-20)).clamp_min(0)
    it = torch.zeros(p.shape, dtype=torch.int32, device=p.device)
    if root:  # the root of a decreasing function, by Newton inside the bracket its signs give
        lo, hi = torch.zeros_like(p), torch.full_like(p, math.inf)
        for _ in range(200):
            d, gap = update(p)
            lo, hi = torch.where(gap > 0, torch.maximum(lo, p), lo), torch.where(gap < 0, torch.minimum(hi, p), hi)
            n = p + d
            out = ~(((n > lo) | (n == 0)) & (n < hi)) & (gap != 0)
            n = torch.where(out, torch.where(hi < math.inf, 0.5 * (lo + hi), 2 * lo + 1e-300), n)
            p = torch.where(gap == 0, p, n)
        it = None
    else:
        live = torch.ones(p.shape, dtype=torch.bool, device=p.device)
        for _ in range(niter):
            d, _ = update(p)
            p = torch.where(live, p + d, p)
            it += live.int()
            live &= ~((d / (p + 1e-10)).abs() < tol)
    a, b = mass(p)
    us = 0.5 * (ul + (pl - p) / (a + 1e-20) + ur - (pr - p) / (b + 1e-20))
    left = us > 0
    ro, po = torch.where(left, rl, rr), torch.where(left, pl, pr)
    shock = ro * ((gamma + 1) * p + (gamma - 1) * po) / ((gamma - 1) * p + (gamma + 1) * po)
    rs = torch.where(p >= po, shock, ro * (p / (po + 1e-20)) ** (1 / gamma)).clamp_min(1e-10)
    cm = torch.maximum(_sound(rl, pl, gamma), _sound(rr, pr, gamma))
    s1, s2 = torch.minimum(ul, ur) - cm > 0, torch.maximum(ul, ur) + cm < 0
    r = torch.where(s1, rl, torch.where(s2, rr, rs))
    u = torch.where(s1, ul, torch.where(s2, ur, us))
    pp = torch.where(s1, pl, torch.where(s2, pr, p))
    t = torch.where(left, ql[2:-1], qr[2:-1])
    return _flux_of(torch.cat([torch.stack([r, u]), t, pp[None]]), gamma), p, it


def _riemann(ql, qr, gamma, name):
    if name == "exact":
        return _riemann_exact(ql, qr, gamma, 10, 1e-6)[0]
    fl, fr = _flux_of(ql, gamma), _flux_of(qr, gamma)
    ul, ur = _cons_of(ql, gamma), _cons_of(qr, gamma)
    sp = 1e-20 / gamma
    rl, rr = ql[0].clamp_min(1e-10), qr[0].clamp_min(1e-10)
    cl, cr = _sound(rl, ql[-1], gamma), _sound(rr, qr[-1], gamma)
    vl, vr = ql[1], qr[1]
    if name == "llf":
        return 0.5 * (fl + fr) - 0.5 * torch.maximum(vl.abs() + cl, vr.abs() + cr) * (ur - ul)
    if name == "hll":
        sl, sr = torch.minimum(vl - cl, vr - cr).clamp_max(0), torch.maximum(vl + cl, vr + cr).clamp_min(0)
        return torch.where(sr - sl < 1e-20, 0.5 * (fl + fr), (sr * fl - sl * fr + sr * sl * (ur - ul)) / (sr - sl))
    pl, pr = torch.maximum(ql[-1], rl * sp), torch.maximum(qr[-1], rr * sp)
    cm = torch.maximum(cl, cr)
    sl, sr = torch.minimum(vl, vr) - cm, torch.maximum(vl, vr) + cm
    a, b = rl * (vl - sl), rr * (sr - vr)
    us = ((b * vr + a * vl + (pl - pr)) / (a + b)).clamp(-1e6, 1e6)
    ps = ((b * pl + a * pr + a * b * (vl - vr)) / (a + b)).clamp_min(0)
    left = us > 0
    q, f0, u0 = torch.where(left, ql, qr), torch.where(left, fl, fr), torch.where(left, ul, ur)
    ro, uo, po, so = (torch.where(left, x, y) for x, y in ((rl, rr), (vl, vr), (pl, pr), (sl, sr)))
    den = torch.where(left, (sl - us).clamp_max(-1e-10), (sr - us).clamp_min(1e-10))
    rs = ro * (so - uo) / den
    star = torch.stack([rs, rs * us] + [rs * t for t in q[2:-1]] + [((so - uo) * u0[-1] - po * uo + ps * us) / den])
    f = torch.where(a + b < 1e-5, 0.5 * (fl + fr), f0 + so * (star - u0))
    return torch.where(sl > 0, fl, torch.where(sr < 0, fr, f))


def _swap(q, d):
    if d == 0:
        return q
    q = q.clone()
    q[[1, 1 + d]] = q[[1 + d, 1]]
    return q


def _ghost1d(u, w, q, side, case, dt, dx, gamma):
    """The 1D build's face state of the neighbour on `side` (w: its conservative state with its own two neighbours)."""
    kind = case["interp"]
    half = 0.5 * _interp(w[0], w[1], w[2], kind)
    far, near = (w[1] - half, w[1] + half) if side == 0 else (w[1] + half, w[1] - half)
    qf, qn = _prim(far, gamma), _prim(near, gamma)
    dq = _slope(qf, qn, q, case["slope"]) if side == 0 else _slope(q, qn, qf, case["slope"])
    return _trace(qn, dq / dx, dt, dx, gamma)


def _step(u, order, dx, case, gamma, cap, edge):
    """One substep of a periodic lattice: u [nvar][cells], x fastest; returns the new state and its dt."""
    nv = u.shape[0]
    nd = nv - 2
    d = u[0].clamp_min(1e-10)
    ekin = 0.5 * d * sum((u[1 + i] / d) ** 2 for i in range(nd))
    p = torch.maximum((u[-1] - ekin) * (gamma - 1), d * 1e-10)
    if cap:
        p = torch.minimum(p, d * 100)
    wave = nd * (gamma * p / d).clamp_min(1e-10).sqrt() + sum((u[1 + i] / d).abs() for i in range(nd))
    dt = min(float((dx / wave).min()) * (math.sqrt(1 + 2 * 0.8 * 1e-4) - 1) / 1e-4, 1e10)
    shape = (nv,) + (edge,) * nd
    U = u.reshape(shape)
    Q = _prim(u, gamma).reshape(shape)
    O = order.reshape(shape[1:])
    new = torch.zeros_like(U)
    own = torch.zeros_like(U)
    before, after = torch.zeros_like(U), torch.zeros_like(U)
    for k in range(nd):
        ax = len(shape) - 1 - k

        def at(a, s, ax=ax):  # the value at the cell s steps up the axis
            return torch.roll(a, -s, ax - (len(shape) - a.dim()))
        q = _swap(Q, k)
        nb = {s: at(q, s) for s in (-2, -1, 1, 2)}
        lo, hi = _trace(q, _slope(nb[-1], q, nb[1], case["slope"]) / dx, dt, dx, gamma)
        for side, s in ((0, -1), (1, 1)):
            if nd == 1:
                w = [at(U, s + o) for o in (-1, 0, 1)]
                glo, ghi = _ghost1d(U, w, q, side, case, dt, dx, gamma)
            else:
                dq = _interp(at(q, s - 1), nb[s], at(q, s + 1), case["interp"]) / (2 * dx)
                glo, ghi = _trace(nb[s], dq, dt, 2 * dx, gamma)
            f = _riemann(ghi, lo, gamma, case["riemann"]) if side == 0 else _riemann(hi, glo, gamma, case["riemann"])
            f = _swap(f, k)
            sign = 1.0 if side == 0 else -1.0
            own = own + sign * f
            # this face's flux leaves the neighbour on its side, at this cell's turn in the loop
            term = -(dt / dx) * sign * at(f, -s) / (1 << nd)
            first = at(O, -s) < O
            before = before + torch.where(first, term, 0.0)
            after = after + torch.where(first, 0.0, term)
    new = U + before + dt / dx * own
    r = new[0].clamp(1e-10, 1e6)
    mom = [torch.minimum(torch.maximum(new[1 + i], -10 * r), 10 * r) for i in range(nd)]
    ek = 0.5 * r * sum((m / r) ** 2 for m in mom)
    floor = r * 1e-10 / (gamma - 1)
    e = torch.where(new[-1] - ek < floor, floor + ek, new[-1])
    new = torch.stack([r] + mom + [torch.minimum(e, r * 1e8)]) + after
    return new.reshape(nv, -1), dt


def _exact_grad(case, seed):
    s = _prepare_grad(case, seed)
    w = torch.from_numpy(_network()).cuda().double()
    x, t = torch.from_numpy(s["x"]).cuda().double(), torch.from_numpy(s["t"]).cuda().double()
    theta = w[:4801].clone().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = theta.split([512, 64, 4096, 64, 64, 1])
    silu = torch.nn.functional.silu
    h = silu(silu(x.t() @ w1.reshape(64, 8).t() + b1) @ w2.reshape(64, 64).t() + b2)
    e = h @ w3 + b3 - t
    (e * e).mean().backward()
    return [theta.grad, float((e * e).sum())]


def exact(case, seed):
    kind = case["kind"]
    if kind == "amr":
        return None  # the whole adaptive run would take minutes
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "exact":
        ql, qr, gam = _stress(case["n"], seed)
        ref = case["mode"] == "reference"
        f, p, it = _riemann_exact(ql, qr, gam, 10, 1e-6, root=not ref)
        return [f, p, it]
    if kind == "boxes":
        fo = _forest(case["nbox"], case["pick"])
        full = torch.zeros(5, fo.f.grid.ncell, device="cuda", dtype=F8)
        u, at = _flow_boxes(fo, seed), 0
        for s in fo.f.specs:
            own = slice(at, at + s.cells)
            full[:, fo.cell[own]] = _step(u[:, own], fo.order[own], s.dx, case, 5.0 / 3.0, False, s.edge)[0]
            at += s.cells
        return full.reshape(-1)
    ndim = 1 if kind == "run1d" else 3
    lay = _uniform(ndim, case.get("nx", 1), case["level"])
    if ndim == 3:
        return _level_full(lay, _step(_flow3d(lay, seed), lay.order, lay.dx, case, 1.4, False, lay.edge)[0])
    u, t, n = _flow1d(lay, seed), 0.0, 0
    if case["tend"] * 7.0 * lay.edge > 60:
        return None  # rounding grows too far on the way (see tolerance)
    while t < case["tend"]:
        u, dt = _step(u, lay.order, lay.dx, case, 1.4, True, lay.edge)
        t, n = t + dt, n + 1
    return [_level_full(lay, u), t, n]
