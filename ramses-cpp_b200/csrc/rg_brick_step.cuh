// rg_brick_step.cuh -- a whole leaf substep of a lattice level in one kernel:
// fluxes, ordered fold, new state, next primitives and CFL candidates.
//
// The face and fold kernels of a level pass 35 doubles a cell through the flux
// scratch (280 bytes written, 280 read back with the event lists; the fold of
// a 128^3 level took 196 us at 5 TB/s for that).  Here a block owns an 8x8x4
// brick, a thread one of its cells: it stages the primitives of the brick and
// a 2-cell halo in shared memory, solves its cell's six Riemann problems and
// leaves each flux in shared memory at the neighbour it refluxes into
// (HydroSolver::godunov_fine, RAMSES-CPP src/solvers/hydro/HydroSolver.cpp:
// 476-482), solves one more problem per thread for the faces through which
// cells outside the brick reflux into it, and after a barrier folds its cell's
// seven updates in the reference's order (the cell's order word, made from
// the plan's event list).  The outside problems are 256 next to 1536 own
// ones; that is what the scratch traffic and a launch cost instead.
//
// 8x8x4 and 256 threads: 46 KB of primitives and 61 KB of fluxes, so that two
// blocks share an SM and one stages or folds while the other solves.  The
// primitives alternate between two arrays (DevStatus::prim_sel: d_prim and the
// flux scratch, which this step leaves unused), since bricks read their
// neighbours' old ones; both hold them in lattice order (x fastest), so a
// brick's rows are read in 16-byte pieces without an index.
#pragma once

#include "rg_brick.cuh"
#include "rg_fold.cuh"

namespace rg {

constexpr int SBZ = 4;                                // brick extent along z
constexpr int SCELLS = BRICK * BRICK * SBZ;           // 256: one thread each
constexpr int SPLANE = BSIDE * BSIDE, SSITES = SPLANE * (SBZ + 2 * BHALO);
constexpr size_t STEP_SMEM = sizeof(double) * (5 * SSITES + 30 * SCELLS);

// Thread of cell (x, y, z) of a brick: half-warps hold rows y and y + 2, which
// are 24 doubles apart and so meet different shared-memory banks.
__device__ __forceinline__ int step_thread(int x, int y, int z) {
    return x | ((y & 2) << 2) | ((y & 1) << 4) | ((y & 4) << 3) | (z << 6);
}

// FLOOR: in the forms with floors; without, false (and nothing done) if the
// brick's values need those.  VOTE: the block looks at the staged states, not
// each cell.
template <int RS, bool BOXED, bool FLOOR, bool VOTE>
__device__ __forceinline__ bool step_brick(const PlanView& P, const BrickGeom& G, const int* __restrict__ lat_id,
                                           const int* __restrict__ lat_ord, int kind, double* __restrict__ prim0,
                                           double* __restrict__ prim1, size_t ncell, double* __restrict__ uold,
                                           double* __restrict__ unew, DevStatus* st, const StepK& K, double dx,
                                           const CflK& F) {
    constexpr int NV = 5;
    extern __shared__ __align__(16) double sq[];  // primitives [NV][SSITES], then incoming fluxes [6][NV][SCELLS]
    double* in = sq + NV * SSITES;
    __shared__ unsigned long long s_min;
    int ex = G.ex, ey = G.ey, ez = G.ez, local = (int)blockIdx.x;
    size_t first = 0;                       // the box's first site
    const size_t pitch = (size_t)P.ncells;  // sites of a plane of primitives (even)
    double dt = st->dt, dtdx = st->dtdx;
    DxDiv D{st->dx, st->inv_dx, st->dx_pow2 != 0};
    unsigned long long* word = &st->dtmin_bits;
    if constexpr (BOXED) {
        // brick_off counts 8^3 bricks, two of this kernel's each
        int lo = 0, hi = G.nbox - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (2 * G.brick_off[mid] <= local) lo = mid;
            else hi = mid - 1;
        }
        local -= 2 * G.brick_off[lo];
        ex = G.ext[3 * lo];
        ey = G.ext[3 * lo + 1];
        ez = G.ext[3 * lo + 2];
        first = (size_t)G.off[lo];
        BoxStep& B = P.boxes[lo];
        dt = B.dt;
        dtdx = B.dtdx;
        dx = B.dx;
        D = DxDiv{B.dx, B.inv_dx, B.dx_pow2 != 0};
        word = &B.dtmin_bits;
    }
    const bool sel = st->prim_sel != 0;
    const double* __restrict__ prim = sel ? prim1 : prim0;
    double* __restrict__ prim_out = sel ? prim0 : prim1;
    const int nbx = ex / BRICK, nby = ey / BRICK;
    const int bx = local % nbx, by = (local / nbx) % nby, bz = local / (nbx * nby);
    const int x0 = bx * BRICK - BHALO, y0 = by * BRICK - BHALO, z0 = bz * SBZ - BHALO;
    Check C;
    // rows of the brick are six pairs of sites, whole pairs on either side of a
    // wrap; a round of the block at a time: the other block of the SM covers
    // its latency, and with the three rounds' loads in flight together the
    // kernel was 3 % slower (registers)
    constexpr int PAIRS = SSITES / 2;
#pragma unroll 1
    for (int k = 0; k < (PAIRS + SCELLS - 1) / SCELLS; ++k) {
        const int t = (int)threadIdx.x + k * SCELLS;
        if (t >= PAIRS) break;
        const int a = 2 * (t % (BSIDE / 2)), b = (t / (BSIDE / 2)) % BSIDE, cz = t / (SPLANE / 2);
        int x = x0 + a, y = y0 + b, z = z0 + cz;
        x = x < 0 ? x + ex : (x >= ex ? x - ex : x);
        y = y < 0 ? y + ey : (y >= ey ? y - ey : y);
        z = z < 0 ? z + ez : (z >= ez ? z - ez : z);
        const size_t g = first + (size_t)x + (size_t)ex * ((size_t)y + (size_t)ey * z);
        double2 v[NV];
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) v[iv] = __ldg(reinterpret_cast<const double2*>(prim + iv * pitch + g));
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) {
            C.up(v[iv].x);
            C.up(v[iv].y);
            reinterpret_cast<double2*>(sq + iv * SSITES)[t] = v[iv];
        }
        if (!FLOOR) {
            C.gas(v[0].x, v[4].x);
            C.gas(v[0].y, v[4].y);
        }
    }
    if (threadIdx.x == 0) s_min = ~0ULL;
    const bool ghost = (kind & KIND_MASK) == K_GHOST;
    const bool fast = __syncthreads_and(!VOTE || (C.top_ok() && (FLOOR || C.gas_ok()))) && ghost && forms_take(D.dx);
    if (!FLOOR && !fast) return false;
    const FastStep S = fast_step(dt, D.dx, D.inv), Sc = fast_step(dt, 2.0 * D.dx, 0.5 * D.inv);
    const int u = threadIdx.x, x = u & 7, y = ((u >> 4) & 1) | ((u >> 2) & 2) | ((u >> 3) & 4), z = u >> 6;
    const int site = (x + BHALO) + BSIDE * (y + BHALO) + SPLANE * (z + BHALO);
    const size_t lsite = (size_t)(bx * BRICK + x) + (size_t)ex * ((size_t)(by * BRICK + y) + (size_t)ey * (bz * SBZ + z));
    const int id = lat_id[first + lsite] - 1;
    int ord = lat_ord[first + lsite];
    unsigned iters = 0;
    double fs[NV];
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) fs[iv] = 0.0;
    // own problems: the flux through the lower face refluxes into the lower neighbour, and so on
#pragma unroll 1
    for (int idim = 0; idim < 3; ++idim) {
        const int stride = idim == 0 ? 1 : (idim == 1 ? BSIDE : SPLANE);
        double f[2][NV];
        unsigned it = 0;
        bool ok = false;
        if (fast) {
            ok = D.pow2 ? brick_dir_fast<RS, true, FLOOR, SSITES, !VOTE>(sq, site, idim, stride, S, Sc, K, f[0], f[1], it)
                        : brick_dir_fast<RS, false, FLOOR, SSITES, !VOTE>(sq, site, idim, stride, S, Sc, K, f[0], f[1], it);
        }
        if (!ok) {
            double g[2 * NV];  // (the call's array lives in memory, the loop's in registers)
            it = brick_dir_plain<RS, SSITES>(sq, site, idim, stride, 0u, ghost, dt, D, K, g);
#pragma unroll
            for (int k = 0; k < 2 * NV; ++k) f[k / NV][k % NV] = g[k];
        }
        iters += it;
        const int c = idim == 0 ? x : (idim == 1 ? y : z), n = idim == 2 ? SBZ : BRICK;
        if (c > 0) {
            double* to = in + (2 * idim) * NV * SCELLS +
                         step_thread(x - (idim == 0), y - (idim == 1), z - (idim == 2));
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) to[iv * SCELLS] = f[0][iv];
        }
        if (c < n - 1) {
            double* to = in + (2 * idim + 1) * NV * SCELLS +
                         step_thread(x + (idim == 0), y + (idim == 1), z + (idim == 2));
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) to[iv * SCELLS] = f[1][iv];
        }
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) fs[iv] = (fs[iv] + f[0][iv]) - f[1][iv];
    }
    // the faces of the cells around the brick towards it: 32 on each x and y
    // side, 64 on each z side, one a thread; the outside cell's slot `side` is
    // the face it shares with the inside cell (cx, cy, cz)
    {
        const int idim = u < 64 ? 0 : (u < 128 ? 1 : 2);
        const int r = u & (idim == 2 ? 127 : 63), half = idim == 2 ? 64 : 32;
        const int side = r < half ? 1 : 0, q = r & (half - 1);
        const int cx = idim == 0 ? (side ? 0 : BRICK - 1) : (q & 7);
        const int cy = idim == 0 ? (q & 7) : (idim == 1 ? (side ? 0 : BRICK - 1) : q >> 3);
        const int cz = idim == 2 ? (side ? 0 : SBZ - 1) : q >> 3;
        const int stride = idim == 0 ? 1 : (idim == 1 ? BSIDE : SPLANE);
        const int inside = (cx + BHALO) + BSIDE * (cy + BHALO) + SPLANE * (cz + BHALO);
        const int outside = inside + (side ? -stride : stride);
        double f[NV];
        bool ok = false;
        if (fast) {
            ok = D.pow2 ? brick_face_fast<RS, true, FLOOR, SSITES, !VOTE>(sq, outside, idim, stride, side, S, Sc, K, f)
                        : brick_face_fast<RS, false, FLOOR, SSITES, !VOTE>(sq, outside, idim, stride, side, S, Sc, K, f);
        }
        if (!ok) {
            double g[NV];
            brick_face_plain<RS, SSITES>(sq, outside, idim, stride, side, ghost, dt, D, K, g);
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) f[iv] = g[iv];
        }
        double* to = in + (2 * idim + side) * NV * SCELLS + step_thread(cx, cy, cz);
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) to[iv * SCELLS] = f[iv];
    }
    double v[NV];
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) v[iv] = uold[iv * ncell + id];
    __syncthreads();
    // the seven updates in loop order (3 bits each: the slot, 7 the cell's own)
    auto reflux = [&](int slot) {
        const double* from = in + slot * NV * SCELLS + u;
        const double w = dtdx * ((slot & 1) ? -1.0 : 1.0);
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) v[iv] = v[iv] - w * from[iv * SCELLS] * 0.125;
    };
    int left = 7;
    for (; (ord & 7) != OWN_SLOT; ord >>= 3, --left) reflux(ord & 7);
    own_update<3>(fs, K.gas, dtdx, v);
    ord >>= 3;
    for (--left; left > 0; ord >>= 3, --left) reflux(ord & 7);
    double q[NV];
    unsigned long long best = ~0ULL, bits;
    if (prim_cfl<3, true, true>(v, q, dx, K.gas, K.smalle, F, &bits)) best = bits;
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        unew[iv * ncell + id] = v[iv];
        uold[iv * ncell + id] = v[iv];
        prim_out[iv * pitch + first + lsite] = q[iv];
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other < best ? other : best;
    }
    if ((u & 31) == 0 && best != ~0ULL) atomicMin(&s_min, best);
    __syncthreads();
    if (u == 0 && s_min != ~0ULL) atomicMin(word, s_min);
    if (RS == RG_RIEMANN_EXACT) {
        unsigned long long wi = iters;
        for (int o = 16; o > 0; o >>= 1) wi += __shfl_xor_sync(0xffffffffu, wi, o);
        if ((u & 31) == 0) {
            atomicAdd(&st->exact_iters, wi);
            atomicAdd(&st->exact_calls, 6ull * 32ull);
        }
    }
    return true;
}

// A brick with gas the forms without floors do not cover, from its staging on.
// Only the HLLC solver has both (us a substep at 128^3, without floors / with
// them everywhere: 454 / 518; a hypersonic flow a third of whose cells are at
// the pressure floor: 686 with both, 1065 with the plain forms behind those
// without floors).  In the others the floors are a few comparisons, and what a
// second copy does to the first one's registers costs more (LLF 456 with both,
// 413 with floors everywhere).
template <int RS, bool BOXED>
__device__ __noinline__ void step_brick_floor(const PlanView& P, BrickGeom G, const int* lat_id, const int* lat_ord,
                                              int kind, double* prim0, double* prim1, size_t ncell, double* uold,
                                              double* unew, DevStatus* st, const StepK& K, double dx, CflK F) {
    step_brick<RS, BOXED, true, false>(P, G, lat_id, lat_ord, kind, prim0, prim1, ncell, uold, unew, st, K, dx, F);
}

template <int RS, bool BOXED>
__global__ void __launch_bounds__(SCELLS, 2)
    k_brick_step(const __grid_constant__ PlanView P, const __grid_constant__ BrickGeom G,
                 const int* __restrict__ lat_id, const int* __restrict__ lat_ord, int kind, double* __restrict__ prim0,
                 double* __restrict__ prim1, size_t ncell, double* __restrict__ uold, double* __restrict__ unew,
                 DevStatus* st, const __grid_constant__ StepK K, double dx, const __grid_constant__ CflK F) {
    if constexpr (RS != RG_RIEMANN_HLLC) {
        step_brick<RS, BOXED, true, true>(P, G, lat_id, lat_ord, kind, prim0, prim1, ncell, uold, unew, st, K, dx, F);
    } else {
        if (!step_brick<RS, BOXED, false, true>(P, G, lat_id, lat_ord, kind, prim0, prim1, ncell, uold, unew, st, K, dx, F))
            step_brick_floor<RS, BOXED>(P, G, lat_id, lat_ord, kind, prim0, prim1, ncell, uold, unew, st, K, dx, F);
    }
}

// CFL candidates and primitives of a lattice level, as k_courant_prim and
// k_courant_prim_boxes form them, the primitives in lattice order.
template <bool BOXED>
__global__ void __launch_bounds__(256)
    k_brick_prefix(PlanView P, BrickGeom G, const int* __restrict__ lat_id, const double* __restrict__ uold,
                   double* __restrict__ prim, size_t ncell, DevStatus* st, double dx,
                   const __grid_constant__ FastGas gas, double smalle, CflK F) {
    constexpr int NV = 5;
    const int lane = threadIdx.x & 31;
    unsigned long long all = ~0ULL;
    for (int base = blockIdx.x * blockDim.x; base < P.ncells; base += gridDim.x * blockDim.x) {
        const int g = base + (int)threadIdx.x;  // (boxes are whole warps: extents are multiples of 8)
        unsigned long long best = ~0ULL, bits;
        int box = 0;
        if (g < P.ncells) {
            if constexpr (BOXED) {
                int lo = 0, hi = G.nbox - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (G.off[mid] <= g) lo = mid;
                    else hi = mid - 1;
                }
                box = lo;
            }
            const size_t id = (size_t)lat_id[g] - 1;
            double u[NV], q[NV];
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) u[iv] = uold[iv * ncell + id];
            if (prim_cfl<3, true, true>(u, q, BOXED ? P.boxes[box].dx : dx, gas, smalle, F, &bits)) best = bits;
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) prim[iv * (size_t)P.ncells + g] = q[iv];
        }
        if constexpr (BOXED) {
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
                best = other < best ? other : best;
            }
            if (lane == 0 && best != ~0ULL) atomicMin(&P.boxes[box].dtmin_bits, best);
        } else {
            all = best < all ? best : all;
        }
    }
    if constexpr (!BOXED) {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, all, o);
            all = other < all ? other : all;
        }
        if (lane == 0 && all != ~0ULL) atomicMin(&st->dtmin_bits, all);
    }
}

template <int RS, bool BOXED>
int launch_brick_step_t(rg_ctx* c, const Plan& P, double dx, int pressure_cap, double cfl) {
    auto kern = k_brick_step<RS, BOXED>;
    static bool attr_set[64] = {};  // per device: the shared-memory opt-in is a function attribute
    const int dev = c->device & 63;
    if (!attr_set[dev]) {
        if (int rc = check_cuda(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STEP_SMEM),
                                "brick step shared memory"))
            return rc;
        attr_set[dev] = true;
    }
    const BrickGeom G{P.lat_e[0], P.lat_e[1], P.lat_e[2], P.nbox, P.bl_ext, P.bl_off, P.bl_brick_off};
    kern<<<P.ncells / SCELLS, SCELLS, STEP_SMEM, c->stream>>>(P.view(), G, P.lat_id, P.lat_ord, P.lat_kind, c->d_prim,
                                                              c->d_flux, (size_t)c->ncell, c->d_uold, c->d_unew,
                                                              c->d_status, step_consts(c), dx, cfl_consts(cfl, pressure_cap));
    return check_cuda(c, cudaGetLastError(), "brick step kernel");
}

}  // namespace rg
