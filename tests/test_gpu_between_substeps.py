"""Calls between two substeps of a level.  A lattice level's substep leaves the
next one's primitives and CFL candidates on the device; whatever else is called
in between, the next substep's bits and dt are the oracle's (one lattice) or
those of an uninterrupted sequence (ensembles)."""
import numpy as np
import pytest

import rg_ensemble as ens
import rg_tree
import rgpu
from refsupport import make_params
from test_gpu_level import bits_equal, ga_of

pytestmark = pytest.mark.gpu

L5 = 5
DX5 = 1.0 / 2 ** L5


class OracleLevel:
    """A level stepped by the oracle."""

    def __init__(self, oracle, g, level, dx, u, **kw):
        self.o, self.ga, self.level, self.dx = oracle, ga_of(g), level, dx
        self.params = make_params(3, **kw)
        self.uold, self.unew = u.copy(), u.copy()

    def step(self):
        dt = self.o.courant(self.ga, 3, 5, self.level, self.dx, 1.4, 0.8, self.uold, pressure_cap=False)
        self.o.set_unew(self.ga, 3, 5, self.level, self.uold, self.unew)
        self.o.godunov_fine(self.ga, self.params, self.level, dt, self.dx, self.uold, self.unew)
        self.o.set_uold(self.ga, 3, 5, self.level, self.uold, self.unew)
        return dt


KW = dict(slope_type=2, riemann="hllc")


def substeps(ctx, how, n):
    """n substeps of the level; their last dt, or None where the call does not give it."""
    if how == "run":
        assert ctx.level_run(L5, DX5, 1e9, max_steps=n)[1] == n
        return None
    for _ in range(n):
        dt = ctx.level_substep(L5, DX5, use_graph=how == "graph", want_dt=True)
    return dt


@pytest.mark.parametrize("how", ["graph", "eager", "run"])
@pytest.mark.parametrize("between", ["output", "output of a coarser level"])
def test_snapshot_between_substeps_of_a_lattice(rgpu_lib, oracle, how, between):
    g = rg_tree.build_uniform(3, L5)
    u = rg_tree.random_state(g, L5, seed=3)
    ref = OracleLevel(oracle, g, L5, DX5, u, **KW)
    ctx = rgpu.Context(make_params(3, **KW), 0)
    try:
        ctx.sync_topology(g)
        ctx.upload_state(u, u)
        got = np.empty_like(u)
        for n in (2, 1, 1, 2, 3, 1):  # the snapshots meet either set of primitives
            for _ in range(n):
                dt = ref.step()
            dt_gpu = substeps(ctx, how, n)
            assert dt_gpu in (None, dt)
            rec = ctx.level_output(L5 if between == "output" else L5 - 1, 3, 5)
            if between == "output":
                ids = np.concatenate([g.ncoarse + ic * g.ngridmax + g.level_octs[L5] for ic in range(8)]) - 1
                assert bits_equal(rec[:, 0].reshape(-1), np.maximum(ref.uold.reshape(5, -1)[0, ids], 1e-10))
            ctx.download_state(uold=got)
            assert bits_equal(got, ref.uold), n
    finally:
        ctx.close()


def forest_run(f, interrupt, steps=6):
    params = rgpu.make_params(3, gamma=f.gamma, courant_factor=0.8, **KW)
    ctx = rgpu.Context(params, 0)
    try:
        ctx.sync_topology(f.grid)
        u = f.initial_state()
        ctx.upload_state(u, u)
        ctx.set_level_boxes(f.level, f.first_oct, f.dx)
        ctx.set_level_lattices(f.level, *f.lattices())
        dts = []
        for k in range(steps):
            ctx.level_substep(f.level, 0.0, use_graph=k % 2 == 0)
            dts.append(ctx.level_box_dt(f.level, f.nbox))
            interrupt(ctx)
        ctx.download_state(uold=u)
        return u, np.array(dts)
    finally:
        ctx.close()


def specs_of(edges, seed=7):
    pool = ens.box_specs(64, seed=seed)
    out = []
    for e in edges:
        out.append(next(s for s in pool if s.edge == e and s not in out))
    return out


def test_snapshot_between_substeps_of_an_ensemble(rgpu_lib):
    f = ens.Forest(specs_of([16, 24, 16]))
    u, dts = forest_run(f, lambda ctx: None)
    v, dts2 = forest_run(f, lambda ctx: ctx.level_output(f.level, 3, 5))
    assert bits_equal(dts, dts2) and bits_equal(u, v)


def two_list_forest():
    """Two boxes, 16^3 and 32^3, the second one's leaf octs in a list of their own after the first one's."""
    f = ens.Forest(specs_of([16, 32]))
    g = f.grid
    octs = g.level_octs[f.level]
    first = int(f.first_oct[1])
    g.nlevelmax = f.level + 1
    g.headl = np.append(g.headl, octs[first]).astype(np.int32)
    g.next[octs[first - 1] - 1] = 0
    g.level_octs[f.level], g.level_octs[f.level + 1] = octs[:first], octs[first:]
    return f


def test_output_that_needs_a_larger_scratch_between_substeps(rgpu_lib):
    """The records of the longer list do not fit the scratch the shorter list's substep left its primitives in."""
    f = two_list_forest()
    ext, lat_id, _ = f.lattices()
    ncell_a = int(ext[0].prod())
    noct = int(f.first_oct[1])
    pos = {int(c): ic * noct + k for ic in range(8) for k, c in
           enumerate(f.grid.ncoarse + ic * f.grid.ngridmax + f.grid.level_octs[f.level])}
    out = []
    for interrupt in (False, True):
        ctx = rgpu.Context(rgpu.make_params(3, gamma=f.gamma, courant_factor=0.8, **KW), 0)
        try:
            ctx.sync_topology(f.grid)
            u = f.initial_state()
            ctx.upload_state(u, u)
            ctx.set_level_boxes(f.level, f.first_oct[:2], f.dx[:1])
            ctx.set_level_lattices(f.level, ext[:1], lat_id[:ncell_a],
                                   np.array([pos[int(c)] for c in lat_id[:ncell_a]], np.int32))
            for k in range(4):
                ctx.level_substep(f.level, 0.0, use_graph=k != 1)
                if interrupt and k == 1:
                    ctx.level_output(f.level + 1, 3, 5)
            ctx.download_state(uold=u)
            out.append((u, ctx.level_box_dt(f.level, 1)))
        finally:
            ctx.close()
    assert bits_equal(out[0][0], out[1][0]) and bits_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("how", ["graph", "eager", "run"])
def test_substep_of_a_refined_level_between_substeps(rgpu_lib, oracle, how):
    """Every cell of level 4 is refined: its substep moves nothing, but takes its own CFL step and primitives."""
    g = rg_tree.build_uniform(3, L5)
    u = rg_tree.random_state(g, L5, seed=5)
    ref = OracleLevel(oracle, g, L5, DX5, u, **KW)
    ctx = rgpu.Context(make_params(3, **KW), 0)
    try:
        ctx.sync_topology(g)
        ctx.upload_state(u, u)
        got = np.empty_like(u)
        for n in (2, 1, 2):
            for _ in range(n):
                dt = ref.step()
            assert substeps(ctx, how, n) in (None, dt)
            assert ctx.level_substep(L5 - 1, 2 * DX5, use_graph=how == "graph", want_dt=True) == 1e10
            ctx.download_state(uold=got)
            assert bits_equal(got, ref.uold), n
    finally:
        ctx.close()


@pytest.mark.parametrize("first", [[0, 2, 3], [0, 0.5, 2, 3], [0, 0.5, 1.25, 2, 3]])
def test_boxes_partitioned_anew(rgpu_lib, first):
    """A partition set after lattices were: the same boxes without them as if they had never been (fewer, as many and
    more boxes; a context that sees only the second partition gives the bits)."""
    f = ens.Forest(specs_of([16, 16, 16]))
    n = int(f.first_oct[1])
    first = np.array([int(x * n) for x in first], np.int32)
    dx = np.full(len(first) - 1, f.dx[0])
    out = []
    for before in (True, False):
        ctx = rgpu.Context(rgpu.make_params(3, gamma=f.gamma, courant_factor=0.8, **KW), 0)
        try:
            ctx.sync_topology(f.grid)
            u = f.initial_state()
            ctx.upload_state(u, u)
            if before:
                ctx.set_level_boxes(f.level, f.first_oct, f.dx)
                ctx.set_level_lattices(f.level, *f.lattices())
                for _ in range(3):
                    ctx.level_substep(f.level, 0.0)
                ctx.upload_state(u, u)
            ctx.set_level_boxes(f.level, first, dx)
            for _ in range(3):
                ctx.level_substep(f.level, 0.0)
            ctx.download_state(uold=u)
            out.append((u, ctx.level_box_dt(f.level, len(dx))))
        finally:
            ctx.close()
    assert bits_equal(out[0][0], out[1][0]) and bits_equal(out[0][1], out[1][1])


def test_refused_lattices_change_nothing(rgpu_lib):
    """Wrong maps between captured substeps are refused; the level goes on with the lattices it has."""
    f = ens.Forest(specs_of([16, 24, 16]))
    ext, lat_id, lat_p = f.lattices()
    swapped, shifted = lat_p.copy(), lat_id.copy()
    swapped[[5, 6]] = swapped[[6, 5]]
    shifted[:16 ** 3] = np.roll(shifted[:16 ** 3].reshape(16, 16, 16), 1, axis=2).reshape(-1)

    def wrong(ctx):
        for e, i, p in ((ext, lat_id, swapped), (ext, shifted, lat_p), (ext[[1, 0, 2]], lat_id, lat_p),
                        (ext + 1, lat_id, lat_p)):
            with pytest.raises(rgpu.RGError):
                ctx.set_level_lattices(f.level, e, i, p)
        assert ctx.face_config(f.level)[0] == shape[0]
    shape = []
    u, dts = forest_run(f, lambda ctx: shape.append(ctx.face_config(f.level)[0]))
    v, dts2 = forest_run(f, wrong)
    assert bits_equal(dts, dts2) and bits_equal(u, v)


def test_lattices_of_boxes_in_another_order(rgpu_lib):
    """The maps of two boxes of one size exchanged: every neighbour matches, but a box's dt and dx are not those of
    the cells listed for it; the same bits as without lattices."""
    f = ens.Forest(specs_of([16, 24, 16]))
    ext, lat_id, lat_p = f.lattices()
    n = 16 ** 3

    def exchanged(a):
        a = a.copy()
        a[:n], a[-n:] = a[-n:].copy(), a[:n].copy()
        return a
    out = []
    for lattices in ((ext, exchanged(lat_id), exchanged(lat_p)), None):
        ctx = rgpu.Context(rgpu.make_params(3, gamma=f.gamma, courant_factor=0.8, **KW), 0)
        try:
            ctx.sync_topology(f.grid)
            u = f.initial_state()
            ctx.upload_state(u, u)
            ctx.set_level_boxes(f.level, f.first_oct, f.dx)
            if lattices:
                ctx.set_level_lattices(f.level, *lattices)
            for _ in range(3):
                ctx.level_substep(f.level, 0.0)
            ctx.download_state(uold=u)
            out.append((u, ctx.level_box_dt(f.level, f.nbox)))
        finally:
            ctx.close()
    assert bits_equal(out[0][0], out[1][0]) and bits_equal(out[0][1], out[1][1])


def fold_ms(ctx, level, dx):
    """Kernel time of a substep's fold: nothing (two events in a row, 3 us) where the substep is one kernel, whose time
    is the face step's; 20 us and more for the fold of 64^3 cells."""
    ctx.set_timing(True)
    ctx.level_substep(level, dx, use_graph=False)
    ctx.level_substep(level, dx, use_graph=False)
    ctx.synchronize()
    face, fold = ctx.kernel_ms()[1:3]
    ctx.set_timing(False)
    assert face > 0.004
    return fold


def test_pinned_shape_outlives_its_plan(rgpu_lib):
    """A pinned lattice level runs the face and fold kernels, also after the plans are rebuilt."""
    g = rg_tree.build_uniform(3, 7)
    u = rg_tree.random_state(g, 7, seed=2)
    ctx = rgpu.Context(make_params(3, **KW), 0)
    try:
        for k in range(3):
            ctx.sync_topology(g)
            ctx.upload_state(u, u)
            ctx.level_substep(7, 1.0 / 128)
            assert (fold_ms(ctx, 7, 1.0 / 128) > 0.008) == (k > 0), k
            if k == 0:
                ctx.set_face_config(7, 10, 1)
                assert fold_ms(ctx, 7, 1.0 / 128) > 0.008
            assert ctx.face_config(7)[0] == 10 or k == 0
    finally:
        ctx.close()
