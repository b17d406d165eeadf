// rg_lattice.cu -- detection of levels that form one complete periodic lattice.
//
// A uniform grid's finest level (the reference's levelmin = levelmax runs, and
// the base level of an AMR run before refinement) holds every cell of an
// Ex x Ey x Ez periodic lattice.  On such a level the plan's neighbour cells
// (AmrGrid::get_nbor_cells, AmrGrid.cpp:402-444) and ghost stencils are the
// lattice neighbours, which lets the brick face kernel (rg_face_brick.cuh)
// stage whole 8^3 bricks of cells in shared memory instead of gathering every
// stencil cell through the plan's index arrays.  Nothing is assumed: the
// lattice is accepted only if, for every cell and interface slot, the plan's
// neighbour id, both ghost-stencil ids and the interface kind equal what the
// lattice gives; otherwise the level keeps the general kernels.
#include <vector>

#include "rg_internal.cuh"

namespace rg {

namespace {

constexpr int LTPB = 256;

// Lattice coordinates of level cell p from its oct's father chain: at every
// level a cell's coordinate is twice its father cell's plus its own bit
// ((ic-1) = ix + 2 iy + 4 iz); coarse cells are numbered x fastest.
// Returns the number of doublings (all cells of a complete level agree).
__device__ int cell_coords(const TreeView& T, const PlanView& P, int p, int* x, int* y, int* z) {
    const int icx = p / P.noct, k = p - icx * P.noct;
    int ig = P.octs[k];
    int cx = icx & 1, cy = (icx >> 1) & 1, cz = (icx >> 2) & 1, scale = 1;
    for (int guard = 0; guard < 40; ++guard) {
        const int fc = T.father[ig - 1];
        scale *= 2;
        if (fc <= 0) return -1;
        if (fc <= T.ncoarse) {
            const int idx = fc - 1;
            cx += scale * (idx % T.nx);
            cy += scale * ((idx / T.nx) % T.ny);
            cz += scale * (idx / (T.nx * T.ny));
            *x = cx;
            *y = cy;
            *z = cz;
            return scale;
        }
        const int j = fc - T.ncoarse - 1, icf = j / T.ngridmax;
        ig = j - icf * T.ngridmax + 1;
        cx += scale * (icf & 1);
        cy += scale * ((icf >> 1) & 1);
        cz += scale * ((icf >> 2) & 1);
    }
    return -1;
}

__global__ void k_lattice_fill(TreeView T, PlanView P, int scale0, int ex, int ey, int ez, int* lat_id, int* lat_p,
                               int* bad) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P.ncells; p += gridDim.x * blockDim.x) {
        int x, y, z;
        const int sc = cell_coords(T, P, p, &x, &y, &z);
        if (sc != scale0 || x < 0 || y < 0 || z < 0 || x >= ex || y >= ey || z >= ez) {
            atomicExch(bad, 1);
            continue;
        }
        const size_t site = (size_t)x + (size_t)ex * ((size_t)y + (size_t)ey * z);
        if (atomicCAS(&lat_p[site], -1, p) != -1) {
            atomicExch(bad, 1);
            continue;
        }
        const int icx = p / P.noct;
        lat_id[site] = T.ncoarse + icx * T.ngridmax + P.octs[p - icx * P.noct];
    }
}

__device__ __forceinline__ int wrap(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// mask != nullptr (a level with refined cells): a refined cell's faces and the
// faces towards one are marked there instead of being of kind kind0.
__global__ void k_lattice_check(TreeView T, PlanView P, int ex, int ey, int ez, const int* __restrict__ lat_id,
                                const int* __restrict__ lat_p, int kind0, uint8_t* mask, int* bad) {
    const size_t n = (size_t)ex * ey * ez;
    for (size_t site = (size_t)blockIdx.x * blockDim.x + threadIdx.x; site < n;
         site += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(site % ex), y = (int)((site / ex) % ey), z = (int)(site / ((size_t)ex * ey));
        const int p = lat_p[site];
        if (p < 0) {
            atomicExch(bad, 1);
            continue;
        }
        const int c = lat_id[site];
        unsigned m = 0;
        if (mask && T.son[c - 1] > 0) {
            mask[site] = LAT_REFINED;
            for (int s = 0; s < 6; ++s)
                if (P.kind[s * (size_t)P.ncells + p] != K_NONE) atomicExch(bad, 1);
            continue;
        }
        for (int s = 0; s < 6; ++s) {
            const int idim = s >> 1, side = s & 1, d = side ? 1 : -1;
            auto at = [&](int off) {
                int xx = x, yy = y, zz = z;
                if (idim == 0) xx = wrap(x + off, ex);
                else if (idim == 1) yy = wrap(y + off, ey);
                else zz = wrap(z + off, ez);
                return lat_id[(size_t)xx + (size_t)ex * ((size_t)yy + (size_t)ey * zz)];
            };
            const int nb = at(d), far = at(2 * d);
            const size_t nc = (size_t)P.ncells;
            const int want_nl = side ? c : far, want_nr = side ? far : c;
            if (mask && P.kind[s * nc + p] == K_ZERO) {
                m |= 1u << s;
                if (P.icn[s * nc + p] != nb) atomicExch(bad, 1);
                continue;
            }
            if (P.icn[s * nc + p] != nb || P.stc[((size_t)s * 2 + 0) * nc + p] != want_nl ||
                P.stc[((size_t)s * 2 + 1) * nc + p] != want_nr || P.kind[s * nc + p] != kind0)
                atomicExch(bad, 1);
        }
        if (mask) mask[site] = (uint8_t)m;
    }
}

// Box lattices supplied by the host (one periodic lattice per ensemble box):
// every site's plan position must hold that site's cell, every plan position
// must appear once, and the plan's neighbours, ghost stencils and kinds must
// be the box lattice's (periodic inside the box).  *other: a site's cell is of
// another box of the partition (boxes alike whose lattices come in another
// order), whose dt and dx the brick kernels would not take.
__global__ void k_box_lattice_check(TreeView T, PlanView P, int nbox, const int* __restrict__ ext,
                                    const int* __restrict__ off, const int* __restrict__ lat_id,
                                    const int* __restrict__ lat_p, int kind0, int* seen, int* bad, int* other) {
    const int n = P.ncells;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        int lo = 0, hi = nbox - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (off[mid] <= g) lo = mid;
            else hi = mid - 1;
        }
        const int b = lo, ex = ext[3 * b], ey = ext[3 * b + 1], ez = ext[3 * b + 2];
        const int site = g - off[b];
        const int x = site % ex, y = (site / ex) % ey, z = site / (ex * ey);
        const int p = lat_p[g], c = lat_id[g];
        if (p < 0 || p >= n || atomicExch(&seen[p], 1) != 0) {
            atomicExch(bad, 1);
            continue;
        }
        const int icx = p / P.noct;
        if (c != T.ncoarse + icx * T.ngridmax + P.octs[p - icx * P.noct]) {
            atomicExch(bad, 1);
            continue;
        }
        if (box_of(P, p) != b) atomicExch(other, 1);
        for (int s = 0; s < 6; ++s) {
            const int idim = s >> 1, side = s & 1, d = side ? 1 : -1;
            auto at = [&](int o) {
                int xx = x, yy = y, zz = z;
                if (idim == 0) xx = wrap(x + o, ex);
                else if (idim == 1) yy = wrap(y + o, ey);
                else zz = wrap(z + o, ez);
                return lat_id[off[b] + xx + ex * (yy + ey * zz)];
            };
            const int nb = at(d), far = at(2 * d);
            const size_t nc = (size_t)n;
            const int want_nl = side ? c : far, want_nr = side ? far : c;
            if (P.icn[s * nc + p] != nb || P.stc[((size_t)s * 2 + 0) * nc + p] != want_nl ||
                P.stc[((size_t)s * 2 + 1) * nc + p] != want_nr || P.kind[s * nc + p] != kind0)
                atomicExch(bad, 1);
        }
    }
}

// Each site's updates in loop order as a word of 3-bit slots (OWN_SLOT: the
// cell's own), from its event list; the list must hold the cell's own update
// and one reflux from each lattice neighbour through the face they share.
// One lattice (nbox 0, extents ex, ey, ez) or one per box.
__global__ void k_lattice_order(PlanView P, int nbox, int ex, int ey, int ez, const int* __restrict__ ext,
                                const int* __restrict__ off, const int* __restrict__ lat_p, int* ord, int* bad) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < P.ncells; g += gridDim.x * blockDim.x) {
        int base = 0;
        if (nbox > 0) {
            int lo = 0, hi = nbox - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (off[mid] <= g) lo = mid;
                else hi = mid - 1;
            }
            base = off[lo];
            ex = ext[3 * lo];
            ey = ext[3 * lo + 1];
            ez = ext[3 * lo + 2];
        }
        const int site = g - base, x = site % ex, y = (site / ex) % ey, z = site / (ex * ey);
        const int p = lat_p[g], a = P.toff[p];
        bool ok = P.toff[p + 1] - a == 7;
        int word = 0, seen = 0;
        for (int e = 0; ok && e < 7; ++e) {
            const int key = P.tev[a + e], slot = key & 7, cp = key >> 3;
            const int ps = (cp & 7) * P.noct + (cp >> 3);
            int xx = x, yy = y, zz = z;
            if (slot != OWN_SLOT) {  // the source whose face `slot` is shared with this cell
                const int d = slot & 1 ? -1 : 1;
                if (slot < 2) xx = wrap(x + d, ex);
                else if (slot < 4) yy = wrap(y + d, ey);
                else zz = wrap(z + d, ez);
            }
            ok = slot != 6 && ps == lat_p[base + xx + ex * (yy + ey * zz)];
            seen |= 1 << slot;
            word |= slot << (3 * e);
        }
        if (!ok || seen != 0xbf) atomicExch(bad, 1);
        ord[g] = word;
    }
}

int lblocks(rg_ctx* c, long long n) {
    long long b = (n + LTPB - 1) / LTPB, cap = (long long)c->sm_count * 16;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

namespace {
// the update order of an accepted lattice (left out, not an error, when the
// event lists are not the lattice's)
int build_order(rg_ctx* c, Plan& P) {
    int* d_bad = nullptr;
    int bad = 1;
    if (P.ntarg != P.ncells) return RG_OK;
    if (int rc = check_cuda(c, dev_alloc(c, &d_bad, sizeof(int)), "lattice order flag")) return rc;
    if (int rc = check_cuda(c, dev_alloc(c, &P.lat_ord, sizeof(int) * (size_t)P.ncells), "lattice order")) return rc;
    cudaMemsetAsync(d_bad, 0, sizeof(int), c->stream);
    k_lattice_order<<<lblocks(c, P.ncells), LTPB, 0, c->stream>>>(P.view(), P.nbox, P.lat_e[0], P.lat_e[1], P.lat_e[2],
                                                                  P.bl_ext, P.bl_off, P.lat_p, P.lat_ord, d_bad);
    cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
    const cudaError_t e = cudaStreamSynchronize(c->stream);
    dev_free(c, d_bad);
    if (bad || e != cudaSuccess) {
        dev_free(c, P.lat_ord);
        P.lat_ord = nullptr;
    }
    return check_cuda(c, e, "lattice order");
}
}  // namespace

// Accepts the level as a lattice (P.lattice = 1, lat_id/lat_p filled) or
// leaves it general.  Synchronises the stream.  Errors are CUDA errors only;
// a level that is not a lattice is not an error.
int build_lattice(rg_ctx* c, Plan& P) {
    P.lattice = 0;
    if (c->params.ndim != 3 || P.level0 || P.ncells == 0 || P.nactive == 0 || P.ilevel < 2) return RG_OK;
    // with refined cells: only levels large enough for the brick face kernel to be timed
    const bool part = P.nactive != P.ncells;
    if (part && P.ncells < (1 << 17)) return RG_OK;
    const long long side = 1LL << (P.ilevel - 1);
    const long long ex = (long long)c->nx * side, ey = (long long)c->ny * side, ez = (long long)c->nz * side;
    if (ex * ey * ez != P.ncells || ex % 8 || ey % 8 || ez % 8) return RG_OK;
    // the interface kind of every face of a uniform leaf level: the first
    // one's; with refined cells it must be the ghost kind
    int8_t kind0 = 0;
    if (int rc = check_cuda(c, cudaMemcpyAsync(&kind0, P.kind, 1, cudaMemcpyDeviceToHost, c->stream), "lattice kind"))
        return rc;
    if (part)
        if (int rc = check_cuda(c, dev_alloc(c, &P.lat_mask, (size_t)P.ncells), "lattice mask")) return rc;
    int* d_bad = nullptr;
    if (int rc = check_cuda(c, dev_alloc(c, &d_bad, sizeof(int)), "lattice flag")) return rc;
    if (int rc = check_cuda(c, dev_alloc(c, &P.lat_id, sizeof(int) * (size_t)P.ncells), "lattice ids")) return rc;
    if (int rc = check_cuda(c, dev_alloc(c, &P.lat_p, sizeof(int) * (size_t)P.ncells), "lattice positions")) return rc;
    cudaMemsetAsync(P.lat_p, 0xff, sizeof(int) * (size_t)P.ncells, c->stream);
    cudaMemsetAsync(d_bad, 0, sizeof(int), c->stream);
    if (int rc = check_cuda(c, cudaStreamSynchronize(c->stream), "lattice kind sync")) return rc;
    const int kd = part ? (K_GHOST | KIND_REFLUX) : kind0;
    if ((kd & KIND_MASK) != K_GHOST && (kd & KIND_MASK) != K_SAME) {
        dev_free(c, d_bad);
        dev_free(c, P.lat_id);
        dev_free(c, P.lat_p);
        dev_free(c, P.lat_mask);
        P.lat_id = P.lat_p = nullptr;
        P.lat_mask = nullptr;
        return RG_OK;
    }
    const int scale0 = (int)side;  // cells per coarse cell and side
    k_lattice_fill<<<lblocks(c, P.ncells), LTPB, 0, c->stream>>>(tree_view(c), P.view(), scale0, (int)ex, (int)ey,
                                                                 (int)ez, P.lat_id, P.lat_p, d_bad);
    k_lattice_check<<<lblocks(c, P.ncells), LTPB, 0, c->stream>>>(tree_view(c), P.view(), (int)ex, (int)ey, (int)ez,
                                                                  P.lat_id, P.lat_p, kd, P.lat_mask, d_bad);
    int bad = 1;
    cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
    const cudaError_t e = cudaStreamSynchronize(c->stream);
    dev_free(c, d_bad);
    if (int rc = check_cuda(c, e, "lattice check")) return rc;
    if (bad) {
        dev_free(c, P.lat_id);
        dev_free(c, P.lat_p);
        dev_free(c, P.lat_mask);
        P.lat_id = P.lat_p = nullptr;
        P.lat_mask = nullptr;
        return RG_OK;
    }
    P.lattice = 1;
    P.lat_e[0] = (int)ex;
    P.lat_e[1] = (int)ey;
    P.lat_e[2] = (int)ez;
    P.lat_kind = kd;
    return part ? RG_OK : build_order(c, P);
}

void drop_lattice(rg_ctx* c, Plan& P) {
    dev_free(c, P.lat_id);
    dev_free(c, P.lat_p);
    dev_free(c, P.lat_ord);
    dev_free(c, P.lat_mask);
    dev_free(c, P.bl_ext);
    dev_free(c, P.bl_off);
    dev_free(c, P.bl_brick_off);
    P.lat_id = P.lat_p = P.lat_ord = P.bl_ext = P.bl_off = P.bl_brick_off = nullptr;
    P.lat_mask = nullptr;
    P.lattice = P.box_lattice = P.bl_nbricks = 0;
}

int set_box_lattices(rg_ctx* c, Plan& P, const int* ext, const int* lat_id, const int* lat_p) {
    const int nbox = P.nbox;
    std::vector<int> hext(ext, ext + 3 * (size_t)nbox), hoff((size_t)nbox), hbrick((size_t)nbox + 1);
    long long sites = 0, bricks = 0;
    for (int b = 0; b < nbox; ++b) {
        const int ex = hext[3 * b], ey = hext[3 * b + 1], ez = hext[3 * b + 2];
        if (ex < 8 || ey < 8 || ez < 8 || ex % 8 || ey % 8 || ez % 8)
            return set_error(c, RG_ERR_ARG, "box " + std::to_string(b) + ": lattice extents must be multiples of 8");
        hoff[(size_t)b] = (int)sites;
        hbrick[(size_t)b] = (int)bricks;
        sites += (long long)ex * ey * ez;
        bricks += (long long)(ex / 8) * (ey / 8) * (ez / 8);
    }
    hbrick[(size_t)nbox] = (int)bricks;
    if (sites != P.ncells) return set_error(c, RG_ERR_ARG, "box lattices do not cover the level's cells once");
    int8_t kind0 = 0;
    // made beside the level's present lattices, which stay as they are when the maps are refused
    struct {
        int *id = nullptr, *p = nullptr, *ext = nullptr, *off = nullptr, *brick = nullptr, *bad = nullptr, *seen = nullptr;
    } N;
    auto drop = [&](int rc) {
        for (int* a : {N.id, N.p, N.ext, N.off, N.brick, N.bad, N.seen}) dev_free(c, a);
        return rc;
    };
    const size_t n = (size_t)P.ncells;
    if (check_cuda(c, dev_alloc(c, &N.bad, 2 * sizeof(int)), "box lattice flags") ||
        check_cuda(c, dev_alloc(c, &N.seen, sizeof(int) * n), "box lattice marks") ||
        check_cuda(c, dev_alloc(c, &N.id, sizeof(int) * n), "box lattice ids") ||
        check_cuda(c, dev_alloc(c, &N.p, sizeof(int) * n), "box lattice positions") ||
        check_cuda(c, dev_alloc(c, &N.ext, sizeof(int) * hext.size()), "box lattice extents") ||
        check_cuda(c, dev_alloc(c, &N.off, sizeof(int) * hoff.size()), "box lattice offsets") ||
        check_cuda(c, dev_alloc(c, &N.brick, sizeof(int) * hbrick.size()), "box lattice bricks"))
        return drop(RG_ERR_NOMEM);
    cudaStream_t s = c->stream;
    cudaMemcpyAsync(&kind0, P.kind, 1, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(N.id, lat_id, sizeof(int) * n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(N.p, lat_p, sizeof(int) * n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(N.ext, hext.data(), sizeof(int) * hext.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(N.off, hoff.data(), sizeof(int) * hoff.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(N.brick, hbrick.data(), sizeof(int) * hbrick.size(), cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(N.seen, 0, sizeof(int) * n, s);
    cudaMemsetAsync(N.bad, 0, 2 * sizeof(int), s);
    if (int rc = check_cuda(c, cudaStreamSynchronize(s), "box lattice upload")) return drop(rc);
    if ((kind0 & KIND_MASK) != K_GHOST && (kind0 & KIND_MASK) != K_SAME)
        return drop(set_error(c, RG_ERR_ARG, "box lattices need a level whose faces are all ghost faces"));
    k_box_lattice_check<<<lblocks(c, P.ncells), LTPB, 0, s>>>(tree_view(c), P.view(), nbox, N.ext, N.off, N.id, N.p,
                                                             kind0, N.seen, N.bad, N.bad + 1);
    int bad[2] = {1, 1};
    cudaMemcpyAsync(bad, N.bad, sizeof(bad), cudaMemcpyDeviceToHost, s);
    if (int rc = check_cuda(c, cudaStreamSynchronize(s), "box lattice check")) return drop(rc);
    if (bad[0]) return drop(set_error(c, RG_ERR_ARG, "box lattices do not match the level's neighbours"));
    // the captured substep names the lattices that go
    if (P.graph) {
        cudaGraphExecDestroy(P.graph);
        P.graph = nullptr;
    }
    drop_lattice(c, P);
    if (bad[1]) return drop(RG_OK);  // accepted, but of no use: the level stays a general one
    dev_free(c, N.bad);
    dev_free(c, N.seen);
    P.lat_id = N.id;
    P.lat_p = N.p;
    P.bl_ext = N.ext;
    P.bl_off = N.off;
    P.bl_brick_off = N.brick;
    P.box_lattice = 1;
    P.bl_nbricks = (int)bricks;
    P.lat_kind = kind0;
    return build_order(c, P);
}

}  // namespace rg
