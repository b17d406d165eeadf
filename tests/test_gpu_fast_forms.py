"""The branch-free forms of the face kernels (csrc/rg_fast.cuh): quotients and
roots against the IEEE operations, and level steps against the oracle on
states that reach each of their limits (operands outside the checked ranges,
floors, zero and tiny numerators, supersonic faces, NaN), in the tiled and the
brick kernel.  Same bits everywhere."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import rg_amr
import rg_tree
import rgpu
from refsupport import make_params
from test_gpu_level import ga_of

pytestmark = pytest.mark.gpu

CSRC = Path(rgpu.__file__).resolve().parent / "csrc"

SOURCE = r"""
#include "rg_fast.cuh"
#include <cstdint>
__device__ uint64_t rnd(uint64_t& s) {
    s += 0x9E3779B97F4A7C15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ double make(uint64_t m, int e) { return __longlong_as_double((long long)((m & 0xfffffffffffffull) | ((uint64_t)(1023 + e) << 52))); }
__global__ void k(int mode, int n, unsigned long long* bad) {
    uint64_t s = (blockIdx.x * blockDim.x + threadIdx.x) * 1000003ull + mode * 77777ull;
    unsigned long long b0 = 0, b1 = 0;
    for (int i = 0; i < n; ++i) {
        uint64_t ra = rnd(s), rb = rnd(s);
        const int ea = (int)(rnd(s) % 1200) - 600, eb = (int)(rnd(s) % 700) - 130;
        if (mode == 1 || mode == 5) rb = ~(rb % 64);          // divisors just below a power of two
        if (mode == 2) { ra = ~(ra % 4096); rb = ~(rb % 4096); }
        if (mode == 3) { ra = ra & 1 ? ~(ra % 4096) : ra % 4096; rb = rb % 4096; }
        const double b = make(rb, eb);
        double a = make(ra, ea);
        if (mode == 4) {                                      // quotients next to a rounding boundary
            const double q = make(ra, 0);
            a = fma(b, q * 0x1p-53, b * q);
        }
        if (mode == 5) a = make(0, ea);                           // powers of two over divisors of mode 1
        if (rb >> 63) a = -a;
        if (rg::rcp_fast(b) != 1.0 / b) ++b0;
        if (rg::div_by(a, b, rg::rcp_fast(b)) != a / b) ++b0;
        double x = make(ra, (ea & 1 ? 1 : 0) + 2 * (ea / 8));
        if (mode == 6) {                                      // roots next to a rounding boundary
            const double h = make(ra, 0);
            x = fma(h, h, h * 0x1p-52);
        }
        if (rg::sqrt_fast(x) != sqrt(x)) ++b1;
    }
    atomicAdd(bad, b0);
    atomicAdd(bad + 1, b1);
}
__global__ void kz(unsigned long long* bad) {                 // zero numerators keep their sign's result
    if (rg::div_by(0.0, 3.0, rg::rcp_fast(3.0)) != 0.0 || signbit(rg::div_by(0.0, 3.0, rg::rcp_fast(3.0)))) ++bad[0];
    if (!signbit(rg::div_by(0.0, -3.0, rg::rcp_fast(-3.0)))) ++bad[0];
}
// the exact solver's two forms on random pairs, odd ones among them
__global__ void ke(int n, int niter, double tol, unsigned long long* bad) {
    uint64_t s = (blockIdx.x * blockDim.x + threadIdx.x) * 99991ull + niter;
    auto uni = [&](double a, double b) { return a + (b - a) * ((rnd(s) >> 11) * 0x1p-53); };
    unsigned long long b0 = 0, plain = 0;
    for (int i = 0; i < n; ++i) {
        double l[5], r[5], f[5], g[5], ps, pg;
        const int odd = rnd(s) % 16;
        for (double* q : {l, r}) {
            q[0] = exp(uni(-12.0, 12.0));
            q[1] = uni(-3.0, 3.0);
            q[2] = uni(-1.0, 1.0);
            q[3] = uni(-1.0, 1.0);
            q[4] = exp(uni(-16.0, 16.0));
        }
        if (odd == 0) for (int k = 0; k < 5; ++k) r[k] = l[k];
        if (odd == 1) { l[1] = -40.0; r[1] = 40.0; }
        if (odd == 2) r[4] = 0.0;
        if (odd == 3) l[4] = -1.0;
        if (odd == 4) r[0] = 1e-13;
        if (odd == 5) l[4] = 1e60;
        if (odd == 6) { l[1] = 50.0; r[1] = 45.0; }
        if (odd == 7) { for (int k = 0; k < 5; ++k) r[k] = l[k]; r[1] += 1e-9; }
        const double gamma = rnd(s) & 1 ? 1.4 : 5.0 / 3.0, smallp = 1e-10 * 1e-10 / gamma;
        const double guess = odd == 8 ? l[4] * 1.1 : -1.0;
        const rg::FastGas G{gamma, gamma - 1.0, 1.0 / (gamma - 1.0), smallp, (gamma + 1.0) / (2.0 * gamma), 1.0 / gamma, 1};
        int it;
        if (!rg::exact_fast<3>(l, r, f, G, niter, tol, guess, &ps, &it)) { ++plain; continue; }
        const int jt = rg::solve_exact_p<3>(l, r, g, gamma, smallp, niter, tol, guess, &pg);
        bool same = it == jt && ps == pg;
        for (int k = 0; k < 5; ++k) same = same && f[k] == g[k];
        if (!same) ++b0;
    }
    atomicAdd(bad, b0);
    atomicAdd(bad + 1, plain);
}
extern "C" int check_exact(int n, int niter, double tol, unsigned long long* out) {
    unsigned long long* d;
    if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
    cudaMemset(d, 0, 16);
    ke<<<592, 128>>>(n, niter, tol, d);
    const int rc = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
extern "C" int check(int mode, int n, unsigned long long* out) {
    unsigned long long* d;
    if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
    cudaMemset(d, 0, 16);
    k<<<592, 256>>>(mode, n, d);
    kz<<<1, 1>>>(d);
    const int rc = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
"""


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    d = tmp_path_factory.mktemp("fast_forms")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-fmad=false", "-shared", "-Xcompiler", "-fPIC", f"-I{CSRC}", "-o", str(d / "t.so"),
                    str(d / "t.cu")], check=True)
    return ctypes.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("mode", range(7))
def test_quotients_and_roots_are_the_ieee_ones(forms, mode):
    bad = (ctypes.c_ulonglong * 2)()
    assert forms.check(mode, 2000, bad) == 0
    assert list(bad) == [0, 0]


@pytest.mark.parametrize("niter,tol", [(10, 1e-6), (100, 1e-14), (1, 1e-6)])
def test_exact_solver_forms_agree(forms, niter, tol):
    """Same iterations, pressure and flux; only the pairs above the checked range take the plain form."""
    out = (ctypes.c_ulonglong * 2)()
    assert forms.check_exact(60, niter, ctypes.c_double(tol), out) == 0
    assert out[0] == 0 and 0 < out[1] < 592 * 128 * 60 // 12


def odd_states(g, level, seed, nan):
    """Random states with patches that reach every limit of the forms."""
    u = rg_tree.random_state(g, level, seed=seed).reshape(5, g.ncell)
    ids = g.cell_ids(level) - 1
    n = len(ids)
    rng = np.random.default_rng(seed)

    def patch(k, m=0.04):
        lo = int(n * k / 12)
        return ids[lo:lo + max(8, int(n * m))]

    def put(cells, rho, v, p):
        u[0, cells] = rho
        for d in range(3):
            u[1 + d, cells] = rho * v[d]
        u[4, cells] = p / 0.4 + 0.5 * rho * sum(x * x for x in v)
    put(patch(0), 1.0, (0.0, 0.0, 0.0), 1.0)                      # at rest: zero slopes, zero numerators
    put(patch(1), 1.0, (0.0, -0.0, 0.0), 1e-5)
    put(patch(2), 2.0, (60.0, -70.0, 80.0), 0.5)                  # supersonic faces
    put(patch(3), 1e-12, (1.0, 0.0, 0.0), 1e-14)                  # below the density floor
    put(patch(4), 1.0, (0.0, 0.0, 0.0), 1e55)                     # above the checked range
    put(patch(5), 1e53, (1e-3, 0.0, 0.0), 1.0)
    put(patch(6), 1.0, (0.0, 0.0, 0.0), 1e-300)                   # pressure floor
    c = patch(7)
    put(c, 1.0, (1e-260, 0.0, 0.0), 1.0)                          # numerators under the checked range
    u[1, c] = rng.uniform(-1e-260, 1e-260, len(c))
    put(patch(8), 1e-7, (0.0, 0.0, 0.0), 1e-9)                    # rc_l + rc_r < 1e-5
    c = patch(9)
    u[4, c] = -u[4, c]                                            # negative energy
    if nan:
        u[rng.integers(0, 5), ids[n // 2]] = np.nan
    return u.reshape(-1)


@pytest.mark.parametrize("level,riem,slope,itype", [(5, "hllc", 1, 1), (6, "hllc", 2, 2), (7, "exact", 1, 1),
                                                    (11, "llf", 8, 3), (13, "hll", 1, 1), (14, "acoustic", 2, 1)])
def test_run_of_a_line_matches_single_substeps(rgpu_lib, level, riem, slope, itype):
    """rg_level_run over a cluster (32 .. 8192 cells; 16 cells and fewer take one block) against the substeps one by
    one: state, primitives' successor step, time and count."""
    g = rg_tree.build_uniform(1, level)
    u = rg_tree.random_state(g, level, seed=level, rho_range=(-0.3, 0.3), p_range=(-0.3, 0.3))
    dx = 1.0 / 2 ** level
    outs = []
    for whole in (True, False):
        ctx = rgpu.Context(make_params(1, slope_type=slope, riemann=riem, interpol_type=itype), 0)
        ctx.sync_topology(g)
        ctx.upload_state(u, u)
        if whole:
            t, n = ctx.level_run(level, dx, 1.0, pressure_cap=True, max_steps=7)
            t, m = ctx.level_run(level, dx, 1.0, t_start=t, pressure_cap=True, max_steps=5)
            n += m
        else:
            t, n = 0.0, 0
            for _ in range(12):
                t += ctx.level_substep(level, dx, pressure_cap=True, use_graph=False, want_dt=True)
                n += 1
        dt = ctx.level_substep(level, dx, pressure_cap=True, use_graph=False, want_dt=True)
        a, b = np.empty_like(u), np.empty_like(u)
        ctx.download_state(a, b)
        outs.append((t, n, dt, a, b))
        ctx.close()
    (t, n, dt, a, b), (t1, n1, dt1, a1, b1) = outs
    assert (t, n, dt) == (t1, n1, dt1)
    assert np.array_equal(a.view(np.int64), a1.view(np.int64)) and np.array_equal(b.view(np.int64), b1.view(np.int64))


def same(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    return np.array_equal(na, nb) and np.array_equal(a[~na].view(np.int64), b[~nb].view(np.int64))


@pytest.mark.parametrize("nan", [False, True])
@pytest.mark.parametrize("variant", [1, 4, 10])
@pytest.mark.parametrize("nx,level,riem,slope,itype", [(1, 5, "hllc", 2, 1), (1, 5, "llf", 1, 2), (3, 4, "hllc", 8, 3),
                                                       (3, 4, "hll", 3, 1), (1, 4, "acoustic", 1, 3),
                                                       (3, 4, "hllc", 2, 0), (1, 4, "hllc", 7, 1)])
def test_level_step_at_the_limits_matches_the_oracle(rgpu_lib, oracle, nx, level, riem, slope, itype, variant, nan):
    g = rg_tree.build_uniform(3, level, nx=nx, ny=nx, nz=nx)
    ga = ga_of(g)
    params = make_params(3, slope_type=slope, riemann=riem, interpol_type=itype)
    ctx = rgpu.Context(params, 0)
    try:
        ctx.sync_topology(g)
        ctx.set_face_config(level, variant, 1)
        dx = 1.0 / (nx * 2 ** level)
        for seed in (1, 2):
            uold = odd_states(g, level, seed, nan)
            unew = uold.copy()
            ctx.upload_state(uold, unew)
            oracle.godunov_fine(ga, params, level, 1e-4, dx, uold.copy(), unew)
            ctx.godunov_level(level, 1e-4, dx)
            got = np.empty_like(unew)
            ctx.download_state(unew=got)
            assert same(got, unew), f"{np.count_nonzero(got != unew)} values differ"
    finally:
        ctx.close()


@pytest.mark.parametrize("nx,level,riem,slope,itype", [(1, 5, "hllc", 2, 1), (3, 4, "llf", 1, 2), (3, 4, "hll", 8, 3),
                                                       (1, 5, "acoustic", 2, 1), (3, 4, "hllc", 4, 1)])
def test_brick_step_at_the_limits_matches_the_oracle(rgpu_lib, oracle, nx, level, riem, slope, itype):
    """Leaf substeps of lattice levels (one kernel a substep, graph and eager mixed, a pinned shape in between)."""
    g = rg_tree.build_uniform(3, level, nx=nx, ny=nx, nz=nx)
    ga = ga_of(g)
    params = make_params(3, slope_type=slope, riemann=riem, interpol_type=itype)
    ctx = rgpu.Context(params, 0)
    try:
        ctx.sync_topology(g)
        dx = 1.0 / (nx * 2 ** level)
        for seed in (3, 4):
            u = odd_states(g, level, seed, False)
            unew = u.copy()
            ctx.upload_state(u, unew)
            for k in range(5):
                if k == 3:
                    ctx.set_face_config(level, 10, 1)  # face and fold kernels from here on
                dt = ctx.level_substep(level, dx, use_graph=k % 2 == 0, want_dt=True)
                assert dt == oracle.courant(ga, 3, 5, level, dx, 1.4, 0.8, u, pressure_cap=False)
                oracle.set_unew(ga, 3, 5, level, u, unew)
                oracle.godunov_fine(ga, params, level, dt, dx, u, unew)
                oracle.set_uold(ga, 3, 5, level, u, unew)
                a, b = np.empty_like(u), np.empty_like(u)
                ctx.download_state(a, b)
                assert same(a, u) and same(b, unew), (seed, k)
    finally:
        ctx.close()


def test_brick_face_kernel_on_a_base_level_with_refined_cells(rgpu_lib):
    """The 64^3 base level of an AMR run (a lattice with refined cells): the brick shapes against the gathering one."""
    ctx = rgpu.Context(make_params(3, slope_type=2, riemann="hllc", courant_factor=0.25), 0)
    try:
        rg_amr.initialize(ctx, 3, 7, 8, 40000, rg_amr.sedov_primitives(3, 7), 1.4, ed=0.1, ep=0.1)
        run = rg_amr.DeviceAmrRun(ctx, nx=1, levelmin=7, nlevelmax=8, cfl=0.25, ed=0.1, ep=0.1)
        for _ in range(3):
            run.coarse_step()
        assert 0 < ctx.cell_updates(7) < 64 ** 3
        got = []
        n = 5 * ctx.tree_sizes()[1]
        for variant in (1, 9, 10):
            ctx.set_face_config(7, variant, 1)
            ctx.set_unew(7)
            ctx.godunov_level(7, 1e-6, 1.0 / 2 ** 7)
            got.append(np.empty(n))
            ctx.download_state(unew=got[-1])
        assert same(got[0], got[1]) and same(got[0], got[2])
    finally:
        ctx.close()


@pytest.mark.parametrize("kw,one", [(dict(slope_type=2), True), (dict(slope_type=0), False), (dict(slope_type=7), False),
                                    (dict(interpol_type=0), False), (dict(interpol_type=4), False),
                                    (dict(riemann="acoustic"), True), (dict(riemann="exact", slope_type=5), False)])
def test_lattice_substeps_take_one_kernel_where_the_forms_apply(rgpu_lib, kw, one):
    """A 64^3 substep's fold time: none in the one-kernel step; slope and interpolation types without branch-free forms
    take the face and fold kernels (there the one kernel was up to 2.7 times slower)."""
    g = rg_tree.build_uniform(3, 7)
    u = rg_tree.random_state(g, 7, seed=1)
    ctx = rgpu.Context(make_params(3, **{**dict(slope_type=1, riemann="hllc"), **kw}), 0)
    try:
        ctx.sync_topology(g)
        ctx.upload_state(u, u)
        ctx.set_timing(True)
        for _ in range(3):
            ctx.level_substep(7, 1.0 / 128, use_graph=False)
        ctx.synchronize()
        assert (ctx.kernel_ms()[2] < 0.008) == one
    finally:
        ctx.close()


def cold_state(g, level, seed):
    """A flow so fast that its thermal energy is lost in the rounding of the total: a third of the cells at the pressure
    floor, negative traced pressures, slow pairs among them."""
    u = g.empty_state().reshape(5, g.ncell)
    x = g.cell_centers(level)
    ids = g.cell_ids(level) - 1
    a = 2 * np.pi * (x + np.random.default_rng(seed).uniform(0, 1, 3))
    rho = np.exp(0.4 * np.sin(a[:, 0] + 2 * a[:, 1]) * np.sin(a[:, 1] + a[:, 2]))
    v = [0.3 * np.sin(a[:, k] + a[:, (k + 1) % 3]) for k in range(3)]
    for k in range(3):
        v[k][:len(ids) // 8] = 0.0                    # gas at rest: nearly equal slow states
    u[0, ids] = rho
    for k in range(3):
        u[1 + k, ids] = rho * v[k]
    u[4, ids] = 1e-12 / 0.4 + 0.5 * rho * sum(w * w for w in v)
    return u.reshape(-1)


@pytest.mark.parametrize("variant", [None, 1, 10])
@pytest.mark.parametrize("nx,level,riem", [(1, 5, "hllc"), (3, 4, "hllc"), (1, 5, "llf"), (3, 4, "hll"), (1, 5, "acoustic")])
def test_cold_gas_matches_the_oracle(rgpu_lib, oracle, nx, level, riem, variant):
    """Pressure floors in the brick step (variant None), the tiled and the brick face kernel."""
    g = rg_tree.build_uniform(3, level, nx=nx, ny=nx, nz=nx)
    ga = ga_of(g)
    params = make_params(3, slope_type=2, riemann=riem)
    ctx = rgpu.Context(params, 0)
    try:
        ctx.sync_topology(g)
        if variant is not None:
            ctx.set_face_config(level, variant, 1)
        dx = 1.0 / (nx * 2 ** level)
        u = cold_state(g, level, 3)
        unew = u.copy()
        ctx.upload_state(u, unew)
        for k in range(4):
            dt = ctx.level_substep(level, dx, use_graph=k % 2 == 0, want_dt=True)
            assert dt == oracle.courant(ga, 3, 5, level, dx, 1.4, 0.8, u, pressure_cap=False)
            oracle.set_unew(ga, 3, 5, level, u, unew)
            oracle.godunov_fine(ga, params, level, dt, dx, u, unew)
            oracle.set_uold(ga, 3, 5, level, u, unew)
            a, b = np.empty_like(u), np.empty_like(u)
            ctx.download_state(a, b)
            assert same(a, u) and same(b, unew), k
        ids = g.cell_ids(level) - 1
        w = u.reshape(5, -1)[:, ids]
        floor = w[4] / w[0] - 0.5 * (w[1:4] ** 2).sum(0) / w[0] ** 2 < 1e-19
        assert floor.mean() > 0.05
    finally:
        ctx.close()
