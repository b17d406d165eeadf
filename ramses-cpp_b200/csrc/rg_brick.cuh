// rg_brick.cuh -- the arithmetic of a cell's faces from a brick of primitives
// staged in shared memory: shared by the brick face kernel (rg_face_brick.cuh)
// and the brick step kernel (rg_brick_step.cuh).
#pragma once

#include "rg_face.cuh"

namespace rg {

constexpr int BRICK = 8, BHALO = 2, BSIDE = BRICK + 2 * BHALO;

// Planes of slots 1..3 for direction idim: rot_swap<3>'s exchange of slot 1
// with slot 1 + idim, applied to where the values are read from, so the
// rotation costs no data movement after the loads.  SITES: sites of a plane.
template <int SITES>
struct BrickPlanes {
    int o1, o2, o3;
    __device__ __forceinline__ explicit BrickPlanes(int idim)
        : o1((1 + idim) * SITES), o2((idim == 1 ? 1 : 2) * SITES), o3((idim == 2 ? 1 : 3) * SITES) {}
    // rotated primitive state of shared-memory site `site`
    __device__ __forceinline__ void load(const double* __restrict__ sq, int site, double* q) const {
        q[0] = sq[site];
        q[1] = sq[o1 + site];
        q[2] = sq[o2 + site];
        q[3] = sq[o3 + site];
        q[4] = sq[4 * SITES + site];
    }
};

// Lattice geometry of a level: one lattice (nbox == 0: extents ex, ey, ez) or
// one lattice per ensemble box (extents ext[3b..3b+2], sites from off[b] in
// the concatenated maps, bricks from brick_off[b]).
struct BrickGeom {
    int ex, ey, ez, nbox;
    const int* ext;
    const int* off;
    const int* brick_off;
};

// The two fluxes of one cell and direction in the plain forms, one trace of the
// cell for both; sides in `none` (bit per side) carry no flux.  put(side, flux)
// takes each as it is known.  Returns the Newton updates.  In line in the kernels without branch-free forms, a call
// where those do not cover a cell: one per direction (a call per face formed
// the cell's trace twice and took 1.3 times the two-kernel step's time where
// every cell went that way), and without the forms with floors in it (what the
// call may overwrite costs the loop around it also where it is not made: with
// them k_brick_step took 474 instead of 434 us at 128^3).
template <int RS, int SITES, class Put>
__device__ __forceinline__ unsigned brick_dir(const double* sq, int site, int idim, int stride, unsigned none, bool ghost,
                                              double dt, const DxDiv& D, const StepK& K, Put put) {
    constexpr int NV = 5;
    const BrickPlanes<SITES> B(idim);
    double qc[NV], ql[NV], qr[NV], qmo[NV], qpo[NV];
    unsigned it = 0;
    B.load(sq, site, qc);
    B.load(sq, site - stride, ql);
    B.load(sq, site + stride, qr);
    own_trace<3>(qc, ql, qr, dt, D, K, qmo, qpo);
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        // neighbour n = c -/+ e, its stencil (n - e, n + e) = (c - 2e, c) / (c, c + 2e)
        double qn[NV], qfar[NV], qm[NV], qp[NV], g[NV];
        if ((none >> side) & 1u) {
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) g[iv] = 0.0;
            put(side, g);
            continue;
        }
        B.load(sq, side ? site + stride : site - stride, qn);
        B.load(sq, side ? site + 2 * stride : site - 2 * stride, qfar);
        const double* qnl = side ? qc : qfar;
        const double* qnr = side ? qfar : qc;
        if (ghost) ghost_trace<3>(qn, qnl, qnr, dt, D, K, qm, qp);
        else own_trace<3>(qn, qnl, qnr, dt, D, K, qm, qp);
        it += side == 0 ? riemann<3, RS>(qm, qpo, g, K) : riemann<3, RS>(qmo, qp, g, K);
        rot_swap<3>(g, idim);
        put(side, g);
    }
    return it;
}
template <int RS, int SITES>
__device__ __noinline__ unsigned brick_dir_plain(const double* sq, int site, int idim, int stride, unsigned none,
                                                 bool ghost, double dt, const DxDiv& D, const StepK& K, double* f) {
    return brick_dir<RS, SITES>(sq, site, idim, stride, none, ghost, dt, D, K, [&](int side, const double* g) {
#pragma unroll
        for (int iv = 0; iv < 5; ++iv) f[side * 5 + iv] = g[iv];
    });
}

// The flux of one cell through one face in the plain forms; `stride` is the
// direction's step between sites.  Returns the Newton updates.
template <int RS, int SITES>
__device__ __noinline__ unsigned brick_face_plain(const double* sq, int site, int idim, int stride, int side,
                                                  bool ghost, double dt, const DxDiv& D, const StepK& K, double* f) {
    constexpr int NV = 5;
    const BrickPlanes<SITES> B(idim);
    const int n = side ? site + stride : site - stride;
    double qc[NV], ql[NV], qr[NV], qn[NV], qmo[NV], qpo[NV], qm[NV], qp[NV];
    B.load(sq, site, qc);
    B.load(sq, site - stride, ql);
    B.load(sq, site + stride, qr);
    own_trace<3>(qc, ql, qr, dt, D, K, qmo, qpo);
    B.load(sq, n, qn);
    B.load(sq, n - stride, ql);
    B.load(sq, n + stride, qr);
    if (ghost) ghost_trace<3>(qn, ql, qr, dt, D, K, qm, qp);
    else own_trace<3>(qn, ql, qr, dt, D, K, qm, qp);
    const unsigned it = side == 0 ? riemann<3, RS>(qm, qpo, f, K) : riemann<3, RS>(qmo, qp, f, K);
    rot_swap<3>(f, idim);
    return it;
}

// The two fluxes of one cell and direction in the branch-free forms (a ghost
// neighbour on both sides, every staged state checked: top_ok, gas_ok; FLOOR:
// with the floors, the states checked here); false: not covered, take the
// plain forms.
template <int RS, bool POW2, bool FLOOR, int SITES, bool CHK = false>
__device__ __forceinline__ bool brick_dir_fast(const double* __restrict__ sq, int site, int idim, int stride,
                                               const FastStep& S, const FastStep& Sc, const StepK& K, double* f0,
                                               double* f1, unsigned& iters) {
    constexpr int NV = 5;
    const BrickPlanes<SITES> B(idim);
    double qc[NV], ql[NV], qr[NV], qfl[NV], qfr[NV], qmo[NV], qpo[NV], qm[NV], qp[NV];
    B.load(sq, site, qc);
    B.load(sq, site - stride, ql);
    B.load(sq, site + stride, qr);
    B.load(sq, site - 2 * stride, qfl);
    B.load(sq, site + 2 * stride, qfr);
    Check C;
    trace_fast<3, POW2, CHK, true, true, FLOOR>(qc, ql, qr, K.own, S, K.gamma, qmo, qpo, C);
    trace_fast<3, POW2, CHK, true, false, FLOOR>(ql, qfl, qc, K.ghost, Sc, K.gamma, qm, nullptr, C);
    trace_fast<3, POW2, CHK, false, true, FLOOR>(qr, qc, qfr, K.ghost, Sc, K.gamma, nullptr, qp, C);
    const bool ok = C.num_ok() && (!CHK || C.top_ok());
    const bool a = riemann_fast<3, RS, FLOOR>(qm, qpo, f0, K, iters), b = riemann_fast<3, RS, FLOOR>(qmo, qp, f1, K, iters);
    rot_swap<3>(f0, idim);
    rot_swap<3>(f1, idim);
    return ok && a && b;
}

// One of them: both face states of both cells are formed and the side's
// chosen, so the two sides share one piece of code.
template <int RS, bool POW2, bool FLOOR, int SITES, bool CHK = false>
__device__ __forceinline__ bool brick_face_fast(const double* __restrict__ sq, int site, int idim, int stride, int side,
                                                const FastStep& S, const FastStep& Sc, const StepK& K, double* f) {
    constexpr int NV = 5;
    const BrickPlanes<SITES> B(idim);
    const int n = side ? site + stride : site - stride;
    double qc[NV], ql[NV], qr[NV], qmo[NV], qpo[NV], qm[NV], qp[NV];
    Check C;
    B.load(sq, site, qc);
    B.load(sq, site - stride, ql);
    B.load(sq, site + stride, qr);
    trace_fast<3, POW2, CHK, true, true, FLOOR>(qc, ql, qr, K.own, S, K.gamma, qmo, qpo, C);
    B.load(sq, n, qc);
    B.load(sq, n - stride, ql);
    B.load(sq, n + stride, qr);
    trace_fast<3, POW2, CHK, true, true, FLOOR>(qc, ql, qr, K.ghost, Sc, K.gamma, qm, qp, C);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        ql[iv] = side ? qmo[iv] : qm[iv];
        qr[iv] = side ? qp[iv] : qpo[iv];
    }
    unsigned it = 0;
    const bool a = riemann_fast<3, RS, FLOOR>(ql, qr, f, K, it);
    rot_swap<3>(f, idim);
    return C.num_ok() && (!CHK || C.top_ok()) && a;
}

}  // namespace rg
