// rg_face_brick.cuh -- face kernel for levels that form one complete periodic
// lattice (detected and verified by rg_lattice.cu), refined cells among them or
// not: the base level of an AMR run is one too (a few of its cells refined).
//
// Same arithmetic and outputs as k_face_tiles (rg_face.cuh): per (cell,
// direction) the own MUSCL-Hancock trace, the two neighbours' face states by
// the ghost (or same-level) branch and the two Riemann fluxes of
// HydroSolver::godunov_fine (RAMSES-CPP src/solvers/hydro/HydroSolver.cpp:
// 93-474); fluxes to the scratch and each cell's own flux sum in the
// reference's (idim, side) order.
//
// A block owns an 8x8x8 brick of cells (on ensemble levels: of one box, whose
// own dt and dx it uses).  It first copies the primitives of
// the brick and a 2-cell periodic halo (12^3 cells, the reach of the own and
// ghost stencils) from HBM into shared memory -- one read of each value per
// brick, through the lattice's id map, instead of per-thread gathers through
// the plan's neighbour and stencil arrays -- and then every thread computes
// all three directions of its cells from shared memory, accumulating the own
// flux sum in registers in slot order.
#pragma once

#include "rg_brick.cuh"

namespace rg {

constexpr int BSITES = BSIDE * BSIDE * BSIDE;
constexpr int BRICK_THREADS = 256;
constexpr size_t BRICK_SMEM = sizeof(double) * 5 * BSITES;  // 69,120 bytes (3D: nvar 5)

// One cell of a brick: its fluxes in the three directions to the scratch, its
// own flux sum in slot order.  FORMS: this instance has the branch-free forms
// (fast: the brick's values allow them); without, the plain ones are in line.
// zero: bit s set where slot s faces a refined cell and carries no flux.
template <int RS, bool FORMS, bool POW2, bool FLOOR, bool CHK>
__device__ __forceinline__ void brick_cell(const double* sq, int site, int p, int nc, bool ghost, bool fast, double dt,
                                           const DxDiv& D, const FastStep& S, const FastStep& Sc, const StepK& K,
                                           unsigned zero, double* __restrict__ flux, double* __restrict__ fsum,
                                           unsigned& iters) {
    constexpr int NV = 5;
    double fs[NV];
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) fs[iv] = 0.0;
#pragma unroll 1
    for (int idim = 0; idim < 3; ++idim) {
        double* out = flux + (size_t)(2 * idim * NV) * nc + p;
        unsigned it = 0;
        const int stride = idim == 0 ? 1 : (idim == 1 ? BSIDE : BSIDE * BSIDE);
        if constexpr (FORMS) {
            const unsigned none = (zero >> (2 * idim)) & 3u;
            double f[2][NV];
            bool ok = false;
            if (fast) ok = brick_dir_fast<RS, POW2, FLOOR, BSITES, CHK>(sq, site, idim, stride, S, Sc, K, f[0], f[1], it);
            if (!ok || none) {
                double g[2 * NV];  // (the call's array lives in memory, the loop's in registers)
                it = brick_dir_plain<RS, BSITES>(sq, site, idim, stride, none, ghost, dt, D, K, g);
#pragma unroll
                for (int k = 0; k < 2 * NV; ++k) f[k / NV][k % NV] = g[k];
            }
#pragma unroll
            for (int k = 0; k < 2 * NV; ++k) out[(size_t)k * nc] = f[k / NV][k % NV];
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) fs[iv] = (fs[iv] + f[0][iv]) - f[1][iv];
        } else {
            // each flux is stored before the next is solved: its registers are free then
            it = brick_dir<RS, BSITES>(sq, site, idim, stride, 0u, ghost, dt, D, K, [&](int side, const double* g) {
#pragma unroll
                for (int iv = 0; iv < NV; ++iv) {
                    out[(size_t)(side * NV + iv) * nc] = g[iv];
                    fs[iv] = side ? fs[iv] - g[iv] : fs[iv] + g[iv];
                }
            });
        }
        iters += it;
    }
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) fsum[(size_t)iv * nc + p] = fs[iv];
}

// The face work of one brick (index `brick` in the level's brick order), by
// the whole block: stage the brick and its halo in sq (shared, [NV][BSITES]),
// then every cell's fluxes and own flux sum.  Newton statistics of the exact
// solver are added to iters / calls.
//
// The cells go through the branch-free forms where the solver's types (FORMS:
// the launch looks), the cell size and the brick's values allow (one vote of
// the block over the staged states); they keep every lane of a warp on one
// straight line, so the two Riemann problems of a direction overlap.  Lanes
// of a half-warp take rows y and y + 2 of the brick: rows are 12 doubles
// apart, so the 16 lanes meet 16 different 8-byte banks.
//
// FLOOR: in the forms with floors; without, false (and nothing done) if the
// level or the brick's values need those or the plain ones.  VOTE: the block
// looks at the staged states, not each cell.
template <int RS, bool BOXED, bool FORMS, bool FLOOR, bool VOTE>
__device__ __forceinline__ bool brick_face(const PlanView& P, const BrickGeom& G, const int* __restrict__ lat_id,
                                           const int* __restrict__ lat_p, const uint8_t* __restrict__ lat_mask,
                                           int kind, const double* __restrict__ prim, size_t ncell,
                                           double* __restrict__ flux, double* __restrict__ fsum, const DevStatus* st, const StepK& K, int brick, double* sq,
                                           unsigned long long& iters, unsigned long long& calls) {
    constexpr int NV = 5;
    int ex = G.ex, ey = G.ey, ez = G.ez, local = brick;
    double dt = st->dt;
    DxDiv D{st->dx, st->inv_dx, st->dx_pow2 != 0};
    if constexpr (BOXED) {
        int lo = 0, hi = G.nbox - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (G.brick_off[mid] <= brick) lo = mid;
            else hi = mid - 1;
        }
        local = brick - G.brick_off[lo];
        ex = G.ext[3 * lo];
        ey = G.ext[3 * lo + 1];
        ez = G.ext[3 * lo + 2];
        lat_id += G.off[lo];
        lat_p += G.off[lo];
        const BoxStep& B = P.boxes[lo];
        dt = B.dt;
        D = DxDiv{B.dx, B.inv_dx, B.dx_pow2 != 0};
    }
    const int nbx = ex / BRICK, nby = ey / BRICK;
    const int bx = local % nbx, by = (local / nbx) % nby, bz = local / (nbx * nby);
    const int x0 = bx * BRICK - BHALO, y0 = by * BRICK - BHALO, z0 = bz * BRICK - BHALO;
    Check C;
    for (int t = threadIdx.x; t < BSITES; t += blockDim.x) {
        const int a = t % BSIDE, b = (t / BSIDE) % BSIDE, cz = t / (BSIDE * BSIDE);
        int x = x0 + a, y = y0 + b, z = z0 + cz;
        x = x < 0 ? x + ex : (x >= ex ? x - ex : x);
        y = y < 0 ? y + ey : (y >= ey ? y - ey : y);
        z = z < 0 ? z + ez : (z >= ez ? z - ez : z);
        const size_t id = (size_t)lat_id[(size_t)x + (size_t)ex * ((size_t)y + (size_t)ey * z)] - 1;
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) {
            const double v = __ldg(prim + iv * ncell + id);
            if (FORMS && VOTE) C.up(v);
            sq[iv * BSITES + t] = v;
        }
        if (FORMS && VOTE && !FLOOR) C.gas(sq[t], sq[4 * BSITES + t]);
    }
    const int nc = P.ncells;
    const bool ghost = (kind & KIND_MASK) == K_GHOST;
    const bool fast = __syncthreads_and(!FORMS || !VOTE || (C.top_ok() && (FLOOR || C.gas_ok()))) && ghost && forms_take(D.dx);
    if (FORMS && !FLOOR && !fast) return false;
    const FastStep S = fast_step(dt, D.dx, D.inv), Sc = fast_step(dt, 2.0 * D.dx, 0.5 * D.inv);
    unsigned it = 0, done = 0;
    for (int u = threadIdx.x; u < BRICK * BRICK * BRICK; u += blockDim.x) {
        const int x = u % BRICK, z = u / (BRICK * BRICK);
        const int y = ((u >> 4) & 1) | ((u >> 2) & 2) | ((u >> 3) & 4);
        const int site = (x + BHALO) + BSIDE * ((y + BHALO) + BSIDE * (z + BHALO));
        const size_t g = (size_t)(bx * BRICK + x) + (size_t)ex * ((size_t)(by * BRICK + y) + (size_t)ey * (bz * BRICK + z));
        const unsigned zero = FORMS && lat_mask ? lat_mask[g] : 0u;
        if (zero & LAT_REFINED) continue;
        const int p = lat_p[g];
        if (!FORMS || D.pow2)
            brick_cell<RS, FORMS, true, FLOOR, !VOTE>(sq, site, p, nc, ghost, fast, dt, D, S, Sc, K, zero, flux, fsum, it);
        else brick_cell<RS, FORMS, false, FLOOR, !VOTE>(sq, site, p, nc, ghost, fast, dt, D, S, Sc, K, zero, flux, fsum, it);
        done += 6 - __popc(zero);
    }
    iters += it;
    calls += done;
    return true;
}

// A brick the forms without floors do not cover, from its staging on.
template <int RS, bool BOXED>
__device__ __noinline__ void brick_face_floor(const PlanView& P, const BrickGeom& G, const int* lat_id, const int* lat_p,
                                              const uint8_t* lat_mask, int kind, const double* prim, size_t ncell,
                                              double* flux, double* fsum, const DevStatus* st, const StepK& K, int brick,
                                              double* sq, unsigned long long* count) {
    unsigned long long iters = 0, calls = 0;
    brick_face<RS, BOXED, true, true, false>(P, G, lat_id, lat_p, lat_mask, kind, prim, ncell, flux, fsum, st, K, brick, sq, iters,
                                      calls);
    count[0] = iters;
    count[1] = calls;
}

template <int RS, int MINB, bool BOXED, bool FORMS>
__global__ void __launch_bounds__(BRICK_THREADS, MINB)
    k_face_brick(const __grid_constant__ PlanView P, const __grid_constant__ BrickGeom G, const int* __restrict__ lat_id, const int* __restrict__ lat_p,
                 const uint8_t* __restrict__ lat_mask, int kind, const double* __restrict__ prim, size_t ncell, double* __restrict__ flux,
                 double* __restrict__ fsum, DevStatus* st, const __grid_constant__ StepK K) {
    extern __shared__ __align__(16) double sq[];  // [NV][BSITES]
    unsigned long long iters = 0, calls = 0;
    if constexpr (FORMS && RS == RG_RIEMANN_HLLC) {
        if (!brick_face<RS, BOXED, true, false, true>(P, G, lat_id, lat_p, lat_mask, kind, prim, ncell, flux, fsum, st, K,
                                                      (int)blockIdx.x, sq, iters, calls)) {
            unsigned long long count[2];
            brick_face_floor<RS, BOXED>(P, G, lat_id, lat_p, lat_mask, kind, prim, ncell, flux, fsum, st, K,
                                        (int)blockIdx.x, sq, count);
            iters = count[0];
            calls = count[1];
        }
    } else {
        brick_face<RS, BOXED, FORMS, true, true>(P, G, lat_id, lat_p, lat_mask, kind, prim, ncell, flux, fsum, st, K,
                                                 (int)blockIdx.x, sq, iters, calls);
    }
    if (RS == RG_RIEMANN_EXACT) {
        for (int o = 16; o > 0; o >>= 1) {
            iters += __shfl_xor_sync(0xffffffffu, iters, o);
            calls += __shfl_xor_sync(0xffffffffu, calls, o);
        }
        if ((threadIdx.x & 31) == 0 && calls) {
            atomicAdd(&st->exact_iters, iters);
            atomicAdd(&st->exact_calls, calls);
        }
    }
}

template <int RS, int MINB, bool BOXED, bool FORMS>
int launch_face_brick_t(rg_ctx* c, const Plan& P, const StepK& K, const double* prim, double* flux, double* fsum) {
    auto kern = k_face_brick<RS, MINB, BOXED, FORMS>;
    static bool attr_set[64] = {};  // per device: the shared-memory opt-in is a function attribute
    const int dev = c->device & 63;
    if (!attr_set[dev]) {
        if (int rc = check_cuda(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)BRICK_SMEM),
                                "brick kernel shared memory"))
            return rc;
        attr_set[dev] = true;
    }
    const BrickGeom G{P.lat_e[0], P.lat_e[1], P.lat_e[2], P.nbox, P.bl_ext, P.bl_off, P.bl_brick_off};
    const int nbricks =
        BOXED ? P.bl_nbricks : (P.lat_e[0] / BRICK) * (P.lat_e[1] / BRICK) * (P.lat_e[2] / BRICK);
    kern<<<nbricks, BRICK_THREADS, BRICK_SMEM, c->stream>>>(P.view(), G, P.lat_id, P.lat_p, P.lat_mask, P.lat_kind, prim,
                                                            (size_t)c->ncell, flux, fsum, c->d_status, K);
    return check_cuda(c, cudaGetLastError(), "brick face kernel");
}

template <int RS, int MINB, bool BOXED = false>
int launch_face_brick(rg_ctx* c, const Plan& P, const StepK& K, const double* prim, double* flux, double* fsum) {
    return K.fast ? launch_face_brick_t<RS, MINB, BOXED, true>(c, P, K, prim, flux, fsum)
                  : launch_face_brick_t<RS, MINB, BOXED, false>(c, P, K, prim, flux, fsum);
}

}  // namespace rg
