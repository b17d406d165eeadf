"""What the runs' main kernels are held to without the reference: the brick step
on ensembles, with the exact solver and on NaN states; the gradient flags
against a restatement of their formula; folds with long targets against the
oracle; and that the kernels meant are the ones that run."""
import numpy as np
import pytest

import rg_amr
import rg_ensemble as ens
import rg_tree
import rgpu
from refsupport import GridArrays, Oracle, make_params
from test_gpu_between_substeps import specs_of
from test_gpu_fast_forms import odd_states, same
from test_gpu_level import EXACT_RTOL, bits_equal, ga_of

pytestmark = pytest.mark.gpu


def kernels_of(fn):
    """Names of the kernels fn launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in p.key_averages())
    if "k_" not in names:
        pytest.skip("the profiler records no kernels here")
    return names


def test_the_kernels_meant_are_the_ones_that_run(rgpu_lib):
    g = rg_tree.build_uniform(3, 5)
    u = rg_tree.random_state(g, 5, seed=1)
    ctx = rgpu.Context(make_params(3, slope_type=2, riemann="hllc"), 0)
    line = rgpu.Context(make_params(1, slope_type=1, riemann="hllc"), 0)
    amr = rgpu.Context(make_params(3, slope_type=2, riemann="hllc", courant_factor=0.25), 0)
    f = ens.Forest(specs_of([16, 24]))
    boxes = rgpu.Context(make_params(3, slope_type=2, riemann="hllc", gamma=f.gamma), 0)
    try:
        ctx.sync_topology(g)
        ctx.upload_state(u, u)

        def substep():
            ctx.level_substep(5, 1.0 / 32, use_graph=False)
            ctx.synchronize()
        assert "k_brick_step" in kernels_of(substep)
        ctx.set_face_config(5, 10, 1)
        names = kernels_of(substep)
        assert "k_face_brick" in names and "k_fold_next" in names and "k_brick_step" not in names
        g1 = rg_tree.build_uniform(1, 8)
        u1 = rg_tree.sod_state(g1, 8, 1.4)
        line.sync_topology(g1)
        line.upload_state(u1, u1)
        assert "k_level_run_line" in kernels_of(lambda: line.level_run(8, 1.0 / 256, 1.0, max_steps=3))
        boxes.sync_topology(f.grid)
        ub = f.initial_state()
        boxes.upload_state(ub, ub)
        boxes.set_level_boxes(f.level, f.first_oct, f.dx)
        boxes.set_level_lattices(f.level, *f.lattices())

        def box_substep():
            boxes.level_substep(f.level, 0.0, use_graph=False)
            boxes.synchronize()
        assert "k_brick_step" in kernels_of(box_substep)
        # the 64^3 base level of an AMR run, some of its cells refined: the brick face kernel
        rg_amr.initialize(amr, 3, 7, 8, 40000, rg_amr.sedov_primitives(3, 7), 1.4, ed=0.1, ep=0.1)
        amr.set_face_config(7, 9, 1)

        def godunov():
            amr.godunov_level(7, 1e-6, 1.0 / 128)
            amr.synchronize()
        assert 0 < amr.count_grids(8) and "k_face_brick" in kernels_of(godunov)
    finally:
        for c in (ctx, line, amr, boxes):
            c.close()


@pytest.mark.parametrize("riem", ["hllc", "llf", "hll"])
def test_ensemble_brick_steps_match_each_box_alone(rgpu_lib, riem):
    """Boxes of 16^3, 24^3 and 32^3 in the one-kernel substep, each against the oracle's run of it alone."""
    f = ens.Forest(specs_of([16, 24, 32, 16], seed=11))
    orc = Oracle()
    ctx = rgpu.Context(rgpu.make_params(3, slope_type=2, riemann=riem, gamma=f.gamma, courant_factor=0.8), 0)
    try:
        ctx.sync_topology(f.grid)
        u = f.initial_state()
        ctx.upload_state(u, u)
        ctx.set_level_boxes(f.level, f.first_oct, f.dx)
        ctx.set_level_lattices(f.level, *f.lattices())
        dts = []
        for k in range(4):
            ctx.level_substep(f.level, 0.0, use_graph=k % 2 == 1)
            dts.append(ctx.level_box_dt(f.level, f.nbox))
        ctx.download_state(uold=u)
    finally:
        ctx.close()
    op = make_params(3, slope_type=2, riemann=riem, gamma=f.gamma)
    for i, (s, b) in enumerate(zip(f.specs, f.boxes)):
        ga = ga_of(b)
        uold = f.box_state(i)
        unew = uold.copy()
        for k in range(4):
            dt = orc.courant(ga, 3, 5, s.level, s.dx, f.gamma, 0.8, uold, pressure_cap=False)
            assert dt == dts[k][i], (i, k)
            orc.set_unew(ga, 3, 5, s.level, uold, unew)
            orc.godunov_fine(ga, op, s.level, dt, s.dx, uold, unew)
            orc.set_uold(ga, 3, 5, s.level, uold, unew)
        assert bits_equal(f.extract(u, i), uold.reshape(5, b.ncell)[:, b.cell_ids(s.level) - 1]), i


@pytest.mark.parametrize("nx,level,riem,slope", [(1, 5, "hllc", 2), (3, 4, "llf", 1), (3, 4, "hll", 8), (1, 5, "hllc", 1)])
def test_brick_step_on_nan_states_matches_the_oracle(rgpu_lib, oracle, nx, level, riem, slope):
    """A NaN value in one cell: its brick's vote, the fold, the clamps and the CFL step."""
    g = rg_tree.build_uniform(3, level, nx=nx, ny=nx, nz=nx)
    ga = ga_of(g)
    params = make_params(3, slope_type=slope, riemann=riem)
    dx = 1.0 / (nx * 2 ** level)
    for seed in (5, 6, 7):
        u = odd_states(g, level, seed, True)
        unew = u.copy()
        ctx = rgpu.Context(params, 0)
        try:
            ctx.sync_topology(g)
            ctx.upload_state(u, unew)
            for k in range(3):
                dt = ctx.level_substep(level, dx, use_graph=k == 1, want_dt=True)
                want = oracle.courant(ga, 3, 5, level, dx, 1.4, 0.8, u, pressure_cap=False)
                assert dt == want or (np.isnan(dt) and np.isnan(want))
                oracle.set_unew(ga, 3, 5, level, u, unew)
                oracle.godunov_fine(ga, params, level, dt, dx, u, unew)
                oracle.set_uold(ga, 3, 5, level, u, unew)
                a, b = np.empty_like(u), np.empty_like(u)
                ctx.download_state(a, b)
                assert same(a, u) and same(b, unew), (seed, k)
        finally:
            ctx.close()


@pytest.mark.parametrize("nx,level", [(1, 5), (3, 4)])
def test_exact_solver_in_the_brick_step(rgpu_lib, oracle, nx, level):
    """Each substep against the oracle's from the same state, and the same bits and Newton updates as the two kernels.
    The solver's pow differs from glibc's by 3e-12 of a flux (EXACT_RTOL); an update is a sum of fluxes times dt / dx,
    each of them below the level's largest value at a CFL factor of 0.8, and may cancel: 3e-12 of that value."""
    g = rg_tree.build_uniform(3, level, nx=nx, ny=nx, nz=nx)
    ga = ga_of(g)
    dx = 1.0 / (nx * 2 ** level)
    u0 = rg_tree.random_state(g, level, seed=9)
    weights = np.random.default_rng(2).normal(0, 0.1, int(rgpu.lib().rg_mlp_nparam())).astype(np.float32)
    for learned in (False, True):
        out = []
        for variant in (None, 1):
            params = make_params(3, slope_type=2, riemann="exact")
            params.exact_guess = 1 if learned else 0
            ctx = rgpu.Context(params, 0)
            try:
                if learned:
                    ctx.mlp_set(weights)
                ctx.sync_topology(g)
                if variant is not None:
                    ctx.set_face_config(level, variant, 1)
                ctx.upload_state(u0, u0)
                u = u0.copy()
                ctx.exact_stats(reset=True)
                for k in range(4):
                    unew = u.copy()
                    dt = ctx.level_substep(level, dx, use_graph=k % 2 == 0, want_dt=True)
                    assert dt == oracle.courant(ga, 3, 5, level, dx, 1.4, 0.8, u, pressure_cap=False)
                    if not learned:
                        oracle.godunov_fine(ga, params, level, dt, dx, u, unew)
                    ctx.download_state(uold=u)
                    assert learned or np.max(np.abs(u - unew)) <= EXACT_RTOL * np.max(np.abs(unew)), k
                out.append((u.copy(), ctx.exact_stats()))
            finally:
                ctx.close()
        assert bits_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


# ---------------------------------------------------------------- gradient flags

def flag_errors(u, edge, gamma):
    """Per lattice site and direction the density and pressure criterion's value (TreeUpdater.cpp:491-535); u [5][e^3]."""
    with np.errstate(all="ignore"):
        u = u.reshape(5, edge, edge, edge)
        d = np.where(u[0] < 1e-10, 1e-10, u[0])
        v2 = 0.0
        for k in range(3):
            v = u[1 + k] / d
            v2 = v2 + v * v
        p = (u[4] - 0.5 * d * v2 - 0.0 - 0.0) * (gamma - 1.0)
        p = np.where(p < d * 1e-10, d * 1e-10, p)
        out = []
        for q in (d, p):
            for axis in (2, 1, 0):
                left, right = np.roll(q, 1, axis), np.roll(q, -1, axis)
                a = np.abs(right - q) / (right + q + 1e-10)
                b = np.abs(q - left) / (q + left + 1e-10)
                out.append(2.0 * np.where(a < b, b, a))
        return np.array(out[:3]).reshape(3, -1), np.array(out[3:]).reshape(3, -1)


@pytest.mark.parametrize("nan", [False, True])
def test_gradient_flags_match_their_formula(rgpu_lib, nan):
    """Thresholds at a cell's own value and one place either side, far outside the division-free tests' range, and each
    criterion alone, over states that reach every limit."""
    level, edge = 5, 16
    g = rg_tree.build_uniform(3, level, ngridmax=3000, nlevelmax=level + 1)
    u = odd_states(g, level, 4, nan)
    ids = g.cell_ids(level) - 1
    ijk = np.rint(g.cell_centers(level) * edge - 0.5).astype(np.int64)
    site = ijk[:, 0] + edge * (ijk[:, 1] + edge * ijk[:, 2])
    lat = np.empty((5, edge ** 3))
    lat[:, site] = u.reshape(5, -1)[:, ids]
    ed_of, ep_of = flag_errors(lat, edge, 1.4)
    rng = np.random.default_rng(1)
    finite = [x[np.isfinite(x) & (x > 0)] for x in (ed_of, ep_of)]
    tests = [(0.1, 0.1), (0.05, -1.0), (-1.0, 0.3), (1e-40, 1.0), (1.0, 1e40), (2.0, 2.0), (0.0, 0.2)]
    for _ in range(6):
        a, b = (float(rng.choice(x)) for x in finite)
        for t in (a, np.nextafter(a, 0.0), np.nextafter(a, 9.0)):
            tests.append((t, -1.0))
        for t in (b, np.nextafter(b, 0.0), np.nextafter(b, 9.0)):
            tests.append((-1.0, t))
    ctx = rgpu.Context(make_params(3, slope_type=1, riemann="hllc"), 0)
    try:
        arrays = rg_tree.tree_arrays(g)
        counts = set()
        for ed, ep in tests:
            ctx.tree_attach(g, arrays, level)
            ctx.upload_state(u, u)
            ctx.flag_fine(level, ed, ep, -1.0, -1.0, 0, 2, 2)
            got = ctx.tree_fetch(arrays)["flag1"][ids]
            want = np.zeros(edge ** 3, bool)
            with np.errstate(invalid="ignore"):
                if ed > 0.0:
                    want |= (ed_of > ed).any(axis=0)
                if ep > 0.0:
                    want |= (ep_of > ep).any(axis=0)
            assert np.array_equal(got != 0, want[site]), (ed, ep)
            counts.add(int(want.sum()))
        assert len(counts) > 8
    finally:
        ctx.close()


# ---------------------------------------------------------------- folds with long targets

def test_folds_of_a_refined_tree_match_the_oracle(rgpu_lib, oracle):
    """Level steps of a tree refined around random cells: coarse cells with fine faces on one to five sides and edges,
    whose targets take tens to hundreds of updates."""
    def ic(xc):
        k = np.floor(xc * 16).astype(np.int64)
        dense = ((k[:, 0] * 73856093) ^ (k[:, 1] * 19349663) ^ (k[:, 2] * 83492791)) % 11 == 0
        rho = np.where(dense, 8.0, 1.0) + 0.01 * np.sin(40 * xc[:, 0])
        return rho, [0.1 * np.sin(9 * xc[:, (d + 1) % 3]) for d in range(3)], 1.0 + 0.3 * np.cos(7 * xc[:, 2])
    params = make_params(3, slope_type=2, riemann="hllc")
    ctx = rgpu.Context(params, 0)
    try:
        rg_amr.initialize(ctx, 3, 4, 6, 30000, ic, 1.4, ed=0.5, ep=-1.0, nexpand=0)
        like = rg_tree.tree_arrays(rg_tree.build_uniform(3, 4, ngridmax=30000, nlevelmax=6))
        a = ctx.tree_fetch(like)
        ngm, ncell = ctx.tree_sizes()
        ga = GridArrays(ncoarse=1, ngridmax=ngm, ncell=ncell, nvar=5, nx=1, ny=1, nz=1, ncpu=1, nboundary=0, nlevelmax=6,
                        son=a["son"], father=a["father"], nbor=a["nbor"], next=a["next"], headl=a["headl"])
        long_targets = 0
        for level in (4, 5, 6):
            assert ctx.count_grids(level) > 0
            dx = 1.0 / 2 ** level
            uold, unew = a["uold"].copy(), a["uold"].copy()
            ctx.upload_state(uold, unew)
            dt = 0.3 * oracle.courant(ga, 3, 5, level, dx, 1.4, 0.8, uold, pressure_cap=False)
            oracle.godunov_fine(ga, params, level, min(dt, 1e-3), dx, uold.copy(), unew)
            ctx.godunov_level(level, min(dt, 1e-3), dx)
            got = np.empty_like(unew)
            ctx.download_state(unew=got)
            assert bits_equal(got, unew), f"level {level}: {np.count_nonzero(got != unew)} values"
            long_targets += ctx.plan_info(level)["nlong"]
        assert long_targets > 20
    finally:
        ctx.close()
