// rg_run1d.cu -- rg_level_run on a 1D level that is one periodic line of
// cells: the whole loop in one launch of one thread-block cluster.
//
// A step of a few thousand cells is a chain of dependent FP64 operations
// (CFL step, traces, Riemann solves, fold, again), so its time is latency and
// what one SM's FP64 pipe can take: in a single block 1024 cells cost 20 us a
// step, each phase through global memory.  Here the line is cut into kCta
// pieces, one SM each; a block keeps its piece's state and primitives in
// shared memory with three cells of each neighbour piece, computes the fluxes
// of its cells and of one more on either side (so no flux travels), and after
// the fold writes its edge cells into the neighbours' copies and its smallest
// CFL candidates into every block's through distributed shared memory: one
// cluster barrier a step.  A (cell, side) pair is one thread's work, lower sides
// first: the warps but the one where the sides meet have one side each.  Same functions on the same operands in the same
// order as the level kernels, so the same bits.
#include <cooperative_groups.h>

#include "rg_fold.cuh"

namespace cg = cooperative_groups;

namespace rg {
namespace {

constexpr int kCta = 8;          // the portable cluster size
constexpr int kLineHalo = 3;     // a cell's new state reaches three cells to either side
constexpr int kLineThreads = 288;  // nine warps: the 260 pairs of a 1024-cell line's piece in one round
constexpr int kLineWarps = kLineThreads / 32;

// Is the level one periodic line in list order?  Site i = 2 k + ic - 1 of the
// list must neighbour i - 1 and i + 1, its ghost stencils must be those of the
// line, both faces ghost faces that reflux, and its updates the three of the
// line in loop order.  *bad counts the cells that differ.
__global__ void k_line_check(TreeView T, PlanView P, int* bad) {
    const int n = P.ncells;
    auto id_at = [&](int i) {
        i = i < 0 ? i + n : (i >= n ? i - n : i);
        return T.ncoarse + (i & 1) * T.ngridmax + P.octs[i >> 1];
    };
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = (i & 1) * P.noct + (i >> 1);
        bool ok = P.icn[p] == id_at(i - 1) && P.icn[(size_t)n + p] == id_at(i + 1);
        ok = ok && P.stc[p] == id_at(i - 2) && P.stc[(size_t)n + p] == id_at(i);
        ok = ok && P.stc[(size_t)2 * n + p] == id_at(i) && P.stc[(size_t)3 * n + p] == id_at(i + 2);
        ok = ok && P.kind[p] == (K_GHOST | KIND_REFLUX) && P.kind[(size_t)n + p] == (K_GHOST | KIND_REFLUX);
        const int a = P.toff[p], l = i > 0 ? i - 1 : n - 1, r = i < n - 1 ? i + 1 : 0;
        ok = ok && P.toff[p + 1] - a == 3;
        if (ok) {
            // (key = loop position * 8 + slot, ascending)
            int want[3] = {l * 8 + 1, i * 8 + OWN_SLOT, r * 8};
            for (int x = 0; x < 2; ++x)
                for (int y = 0; y < 2 - x; ++y)
                    if (want[y] > want[y + 1]) {
                        const int w = want[y];
                        want[y] = want[y + 1];
                        want[y + 1] = w;
                    }
            for (int e = 0; e < 3; ++e) ok = ok && P.tev[a + e] == want[e];
        }
        if (!ok) atomicAdd(bad, 1);
    }
}

// Shared memory of a block: two copies of the piece with its halo (state and
// primitives), the fluxes, the CFL candidates of every warp of the cluster.
struct LineSmem {
    double *u, *q, *f;
    unsigned long long* cfl;
    int pitch, fp;  // sites of a copy, of the flux arrays
    __device__ LineSmem(double* base, int m) : pitch(m + 2 * kLineHalo), fp(m + 2) {
        cfl = reinterpret_cast<unsigned long long*>(base);
        u = base + 2 * kCta * kLineWarps;
        q = u + 2 * 3 * pitch;
        f = q + 2 * 3 * pitch;
    }
};
size_t line_smem(int m) {
    return sizeof(double) * (2 * kCta * kLineWarps + 2 * 2 * 3 * (size_t)(m + 2 * kLineHalo) + 2 * 3 * (size_t)(m + 2));
}

// The flux of one (cell, side) pair in the branch-free forms (conservative
// interpolation of the ghost states): ghost_1d_states, own_trace and the
// solver on the same operands.  False: not covered, take the plain forms.
template <int RS, bool POW2>
__device__ __forceinline__ bool line_flux_fast(const double* uc, const double* ul, const double* ur, const double* qc,
                                               const double* ql, const double* qr, int side, const FastStep& S,
                                               const StepK& K, double* f, unsigned& it) {
    constexpr int NV = 3;
    Check C;
    C.gas(qc[0], qc[2]);
    double qmo[NV], qpo[NV], far[NV], near[NV], qf[NV], qn[NV], qa[NV], qb[NV], qm[NV], qp[NV];
    trace_fast<1, POW2, true, true, true>(qc, ql, qr, K.own, S, K.gamma, qmo, qpo, C);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        const double h = 0.5 * limited<true>(ul[iv], uc[iv], ur[iv], K.ghost, C);
        far[iv] = side ? uc[iv] + h : uc[iv] - h;
        near[iv] = side ? uc[iv] - h : uc[iv] + h;
        C.up(far[iv]);
        C.up(near[iv]);
    }
    auto prim = [&](const double* u, double* q) {  // ctoprim with the branch-free reciprocal
        const double d = smax(u[0], 1e-10), o = div_by(1.0, d, rcp_fast(d));
        q[0] = d;
        q[1] = u[1] * o;
        q[2] = K.gas.gm1 * d * smax(u[2] * o - (0.0 + 0.5 * q[1] * q[1]) - 0.0, K.smalle);
    };
    prim(far, qf);
    prim(near, qn);
    C.gas(qn[0], qn[2]);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        const double l = side ? qn[iv] - qc[iv] : qn[iv] - qf[iv], r = side ? qf[iv] - qn[iv] : qc[iv] - qn[iv];
        qa[iv] = qn[iv] - l;
        qb[iv] = qn[iv] + r;
    }
    trace_fast<1, POW2, true, true, true>(qn, qa, qb, K.own, S, K.gamma, qm, qp, C);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        qa[iv] = side ? qmo[iv] : qm[iv];
        qb[iv] = side ? qp[iv] : qpo[iv];
    }
    const bool ok = riemann_fast<1, RS>(qa, qb, f, K, it);
    return ok && C.top_ok() && C.num_ok() && C.gas_ok();
}

template <int RS>
__device__ __noinline__ int line_flux_plain(const double* uc, const double* ul, const double* ur, const double* qc,
                                            const double* ql, const double* qr, int side, double dt, const DxDiv& D,
                                            const StepK& K, double* f) {
    constexpr int NV = 3;
    double qmo[NV], qpo[NV], qm[NV], qp[NV];
    own_trace<1>(qc, ql, qr, dt, D, K, qmo, qpo);
    ghost_1d_states(uc, ul, ur, side, qc, dt, D, K, qm, qp);
    return side == 0 ? riemann<1, RS>(qm, qpo, f, K) : riemann<1, RS>(qmo, qp, f, K);
}

template <int RS>
__global__ void __cluster_dims__(kCta, 1, 1) __launch_bounds__(kLineThreads, 1)
    k_level_run_line(TreeView T, PlanView P, double* __restrict__ uold, double* __restrict__ unew,
                     double* __restrict__ prim, DevStatus* st, const __grid_constant__ StepK K, double dx, CflK F,
                     double dt_start, double t_end, long long max_steps) {
    constexpr int NV = 3;
    extern __shared__ __align__(16) double smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), m = P.ncells / kCta, base = rank * m, n = P.ncells;
    const size_t ncell = (size_t)T.ncell;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    LineSmem S(smem, m);
    auto id_at = [&](int i) {
        i = i < 0 ? i + n : (i >= n ? i - n : i);
        return T.ncoarse + (i & 1) * T.ngridmax + P.octs[i >> 1];
    };
    for (int j = threadIdx.x; j < S.pitch; j += blockDim.x) {
        const int id = id_at(base + j - kLineHalo);
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) {
            S.u[iv * S.pitch + j] = uold[(size_t)iv * ncell + id - 1];
            S.q[iv * S.pitch + j] = prim[(size_t)iv * ncell + id - 1];
        }
    }
    const double inv = 1.0 / dx;
    const DxDiv D{dx, inv, is_pow2_with_normal_inverse(dx, inv)};
    const bool fast = K.fast && K.interpol_var == 0 && forms_take(dx);
    const unsigned long long start_bits = (unsigned long long)__double_as_longlong(dt_start);
    unsigned long long word = st->dtmin_bits;
    double t = st->run_t, dt = 0.0;
    long long steps = st->run_steps;
    unsigned iters = 0, calls = 0;
    int cur = 0;
    cluster.sync();  // every piece is there before an edge is written
    for (long long guard = 0; guard < max_steps; ++guard) {
        dt = __longlong_as_double((long long)word);
        const double dtdx = dt / dx;
        const FastStep fs2 = fast_step(dt, dx, inv);
        const double* u = S.u + cur * NV * S.pitch;
        const double* q = S.q + cur * NV * S.pitch;
        // fluxes of cells -1 .. m of the piece, lower faces first
        for (int w = threadIdx.x; w < 2 * S.fp; w += blockDim.x) {
            const int side = w >= S.fp, jj = w - side * S.fp, c = jj - 1 + kLineHalo;
            double qc[NV], ql[NV], qr[NV], ul[NV], uc[NV], ur[NV], f[NV];
            const int nb = side ? c + 1 : c - 1;
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) {
                qc[iv] = q[iv * S.pitch + c];
                ql[iv] = q[iv * S.pitch + c - 1];
                qr[iv] = q[iv * S.pitch + c + 1];
                ul[iv] = u[iv * S.pitch + nb - 1];
                uc[iv] = u[iv * S.pitch + nb];
                ur[iv] = u[iv * S.pitch + nb + 1];
            }
            unsigned it = 0;
            bool ok = false;
            if (fast)
                ok = D.pow2 ? line_flux_fast<RS, true>(uc, ul, ur, qc, ql, qr, side, fs2, K, f, it)
                            : line_flux_fast<RS, false>(uc, ul, ur, qc, ql, qr, side, fs2, K, f, it);
            if (!ok) {
                // (copies: the call's arrays live in memory, the loop's in registers)
                double a[7][NV];
#pragma unroll
                for (int iv = 0; iv < NV; ++iv) {
                    a[0][iv] = uc[iv];
                    a[1][iv] = ul[iv];
                    a[2][iv] = ur[iv];
                    a[3][iv] = qc[iv];
                    a[4][iv] = ql[iv];
                    a[5][iv] = qr[iv];
                }
                it = line_flux_plain<RS>(a[0], a[1], a[2], a[3], a[4], a[5], side, dt, D, K, a[6]);
#pragma unroll
                for (int iv = 0; iv < NV; ++iv) f[iv] = a[6][iv];
            }
            if (RS == RG_RIEMANN_EXACT && jj >= 1 && jj <= m) {
                iters += it;
                ++calls;
            }
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) S.f[(side * NV + iv) * S.fp + jj] = f[iv];
        }
        __syncthreads();
        // ordered fold, next primitives and CFL candidates
        const int nxt = cur ^ 1;
        double* un = S.u + nxt * NV * S.pitch;
        double* qn = S.q + nxt * NV * S.pitch;
        unsigned long long best = ~0ULL;
        for (int j = threadIdx.x; j < m; j += blockDim.x) {
            const int i = base + j;
            double v[NV], fs[NV], fl[NV], fr[NV], qq[NV];
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) {
                v[iv] = u[iv * S.pitch + j + kLineHalo];
                fs[iv] = (0.0 + S.f[iv * S.fp + j + 1]) - S.f[(NV + iv) * S.fp + j + 1];
                fl[iv] = dtdx * -1.0 * S.f[(NV + iv) * S.fp + j] * 0.5;  // the left cell's upper face
                fr[iv] = dtdx * 1.0 * S.f[iv * S.fp + j + 2] * 0.5;      // the right cell's lower face
            }
            // loop order: left, own, right; the two end cells meet the line's other end first or last
            auto sub = [&](const double* x) {
#pragma unroll
                for (int iv = 0; iv < NV; ++iv) v[iv] = v[iv] - x[iv];
            };
            if (i == n - 1) sub(fr);
            if (i > 0) sub(fl);
            own_update<1>(fs, K.gas, dtdx, v);
            if (i < n - 1) sub(fr);
            if (i == 0) sub(fl);
            unsigned long long bits;
            if (prim_cfl<1, true, true>(v, qq, dx, K.gas, K.smalle, F, &bits) && bits < best) best = bits;
            // into this piece and, at its edges, the neighbours' copies
            auto put = [&](double* ub, double* qb, int at) {
#pragma unroll
                for (int iv = 0; iv < NV; ++iv) {
                    ub[iv * S.pitch + at] = v[iv];
                    qb[iv * S.pitch + at] = qq[iv];
                }
            };
            put(un, qn, j + kLineHalo);
            if (j < kLineHalo) {
                const int to = (rank + kCta - 1) % kCta;
                put(cluster.map_shared_rank(un, to), cluster.map_shared_rank(qn, to), m + kLineHalo + j);
            }
            if (j >= m - kLineHalo) {
                const int to = (rank + 1) % kCta;
                put(cluster.map_shared_rank(un, to), cluster.map_shared_rank(qn, to), j - (m - kLineHalo));
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other < best ? other : best;
        }
        if (lane < kCta)
            cluster.map_shared_rank(S.cfl + nxt * kCta * kLineWarps, lane)[rank * kLineWarps + warp] = best;
        t = t + dt;
        ++steps;
        cluster.sync();
        cur = nxt;
        word = start_bits;
        for (int k = lane; k < kCta * kLineWarps; k += 32) {
            const unsigned long long x = S.cfl[cur * kCta * kLineWarps + k];
            word = x < word ? x : word;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, word, o);
            word = other < word ? other : word;
        }
        if (!(t < t_end && steps < max_steps)) break;  // the same clock in every thread
    }
    // (no block leaves, or is written to, after the last barrier)
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const int id = id_at(base + j);
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) {
            const double v = S.u[(cur * NV + iv) * S.pitch + j + kLineHalo];
            uold[(size_t)iv * ncell + id - 1] = v;
            unew[(size_t)iv * ncell + id - 1] = v;
            prim[(size_t)iv * ncell + id - 1] = S.q[(cur * NV + iv) * S.pitch + j + kLineHalo];
        }
    }
    if (RS == RG_RIEMANN_EXACT && calls) {
        atomicAdd(&st->exact_iters, (unsigned long long)iters);
        atomicAdd(&st->exact_calls, (unsigned long long)calls);
    }
    if (rank == 0 && threadIdx.x == 0) {
        st->dt = dt;
        st->dx = dx;
        st->dtdx = dt / dx;
        st->inv_dx = inv;
        st->dx_pow2 = D.pow2 ? 1 : 0;
        st->dtmin_bits = word;
        st->run_t = t;
        st->run_steps = steps;
    }
}

template <int RS>
int launch_line(rg_ctx* c, const Plan& P, double dx, int pressure_cap, double t_end, long long max_steps) {
    const StepK K = step_consts(c);
    auto kern = k_level_run_line<RS>;
    const size_t smem = line_smem(P.ncells / kCta);
    // the kernel's limit is the longest line's: threads with lines of several sizes share it
    if (int rc = check_cuda(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)line_smem(kLineCells / kCta)),
                            "line run shared memory"))
        return rc;
    kern<<<kCta, kLineThreads, smem, c->stream>>>(tree_view(c), P.view(), c->d_uold, c->d_unew, c->d_prim, c->d_status,
                                                  K, dx, cfl_consts(c->params.courant_factor, pressure_cap),
                                                  c->params.boxlen / 1e-10, t_end, max_steps);
    return check_cuda(c, cudaGetLastError(), "line run kernel");
}

}  // namespace

int line_check(rg_ctx* c, Plan& P) {
    if (P.line >= 0) return RG_OK;
    P.line = 0;
    if (c->params.ndim != 1 || P.level0 || P.nbox > 0 || P.ncells % kCta || P.ncells < kCta * kLineHalo ||
        P.ncells > kLineCells || P.ntarg != P.ncells)
        return RG_OK;
    int* bad = nullptr;
    int h = 1;
    if (int rc = check_cuda(c, dev_alloc(c, &bad, sizeof(int)), "line check")) return rc;
    cudaMemsetAsync(bad, 0, sizeof(int), c->stream);
    k_line_check<<<(P.ncells + 255) / 256, 256, 0, c->stream>>>(tree_view(c), P.view(), bad);
    cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
    const int rc = check_cuda(c, cudaStreamSynchronize(c->stream), "line check");
    dev_free(c, bad);
    if (rc) return rc;
    P.line = h == 0;
    return RG_OK;
}

int launch_run_line(rg_ctx* c, const Plan& P, double dx, int pressure_cap, double t_end, long long max_steps) {
    switch (c->params.riemann) {
        case RG_RIEMANN_HLLC: return launch_line<RG_RIEMANN_HLLC>(c, P, dx, pressure_cap, t_end, max_steps);
        case RG_RIEMANN_HLL: return launch_line<RG_RIEMANN_HLL>(c, P, dx, pressure_cap, t_end, max_steps);
        case RG_RIEMANN_EXACT: return launch_line<RG_RIEMANN_EXACT>(c, P, dx, pressure_cap, t_end, max_steps);
        case RG_RIEMANN_ACOUSTIC: return launch_line<RG_RIEMANN_ACOUSTIC>(c, P, dx, pressure_cap, t_end, max_steps);
        default: return launch_line<RG_RIEMANN_LLF>(c, P, dx, pressure_cap, t_end, max_steps);
    }
}

}  // namespace rg
