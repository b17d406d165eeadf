// rg_brick_step.cu -- instantiation and launch of the brick step kernel.
#include <algorithm>

#include "rg_brick_step.cuh"

namespace rg {

int launch_brick_prefix(rg_ctx* c, const Plan& P, double dx, int pressure_cap, double cfl) {
    const StepK K = step_consts(c);
    const BrickGeom G{P.lat_e[0], P.lat_e[1], P.lat_e[2], P.nbox, P.bl_ext, P.bl_off, P.bl_brick_off};
    const int blocks = std::min((P.ncells + 255) / 256, c->sm_count * 32);
    if (P.nbox > 0)
        k_brick_prefix<true><<<blocks, 256, 0, c->stream>>>(P.view(), G, P.lat_id, c->d_uold, c->d_prim, (size_t)c->ncell,
                                                            c->d_status, dx, K.gas, K.smalle, cfl_consts(cfl, pressure_cap));
    else
        k_brick_prefix<false><<<blocks, 256, 0, c->stream>>>(P.view(), G, P.lat_id, c->d_uold, c->d_prim, (size_t)c->ncell,
                                                             c->d_status, dx, K.gas, K.smalle, cfl_consts(cfl, pressure_cap));
    return check_cuda(c, cudaGetLastError(), "brick step primitives");
}

int launch_brick_step(rg_ctx* c, const Plan& P, double dx, int pressure_cap, double cfl) {
#define RG_STEP_CASE(rs)                                                                       \
    return P.nbox > 0 ? launch_brick_step_t<rs, true>(c, P, dx, pressure_cap, cfl)            \
                      : launch_brick_step_t<rs, false>(c, P, dx, pressure_cap, cfl)
    switch (c->params.riemann) {
        case RG_RIEMANN_HLLC: RG_STEP_CASE(RG_RIEMANN_HLLC);
        case RG_RIEMANN_HLL: RG_STEP_CASE(RG_RIEMANN_HLL);
        case RG_RIEMANN_EXACT: RG_STEP_CASE(RG_RIEMANN_EXACT);
        case RG_RIEMANN_ACOUSTIC: RG_STEP_CASE(RG_RIEMANN_ACOUSTIC);
        default: RG_STEP_CASE(RG_RIEMANN_LLF);
    }
#undef RG_STEP_CASE
}

}  // namespace rg
