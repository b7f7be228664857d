// FP64 core kernels of the SHAPE B200 engine: model realization, view
// transforms, facet binning, chi-square reductions, lightcurve splines, sky
// frames and the evaluation summary. (Shading, shadows and photometry of a
// pixel belong to the raster, raster_impl.cuh.)
//
// This translation unit is compiled with -fmad=false: the realization, the
// view transforms and the facet bounding boxes must reproduce the reference
// CPU arithmetic bit for bit (no a*b+c contraction), because they decide
// which POS pixels each facet covers. Expressions keep the reference's
// association order; sums that the reference starts from a literal 0.0
// (cotrans, src/util/cotrans.c; mmmul) start from 0.0 here as well.
#include <algorithm>
#include <cfloat>
#include <climits>

#include "kernels.h"
#include "posmask_dev.cuh"

namespace shape {

namespace {

constexpr double SMALLVAL = SHAPE_SMALLVAL;
constexpr double HUGENUMBER = SHAPE_HUGENUMBER;

__device__ inline double dmin_(double a, double b) { return (a < b) ? a : b; }
__device__ inline double dmax_(double a, double b) { return (a > b) ? a : b; }
__device__ inline int clamp_lo(double v) { return (v < (double)INT_MIN) ? INT_MIN : (int)v; }
__device__ inline int clamp_hi(double v) { return (v > (double)INT_MAX) ? INT_MAX : (int)v; }

// ---------------------------------------------------------------- realize

// x = scale * (u*r + a)  (src/shape/realize_mod.c:471-479)
// Several components (vcomp and cxf non-null): vertex i takes its
// component's scale factors, then the component's rotation (comp.m, when
// its rotation offsets are not all zero) and translation (when its offsets
// are not all zero), as realize_mod does (src/shape/realize_mod.c:474-512).
// cxf holds per component m (9, row-major), off (3) and the two flags.
// P: where the deviations and scale factors are read (r(i), scale(k)).
struct ArrayParams {
    const double *__restrict__ rv;
    const double *__restrict__ sv;
    __device__ double r(int i) const { return rv[i]; }
    __device__ double scale(int k) const { return sv[k]; }
};
template <typename P>
__device__ inline double4 realize_vertex(int i, const double *__restrict__ a, const double *__restrict__ u, const P &par,
                                         const int *__restrict__ vcomp, const double *__restrict__ cxf)
{
    const int c = vcomp ? vcomp[i] : 0;
    double ri = par.r(i);
    double x0 = par.scale(3 * c + 0) * (u[3 * i + 0] * ri + a[3 * i + 0]);
    double x1 = par.scale(3 * c + 1) * (u[3 * i + 1] * ri + a[3 * i + 1]);
    double x2 = par.scale(3 * c + 2) * (u[3 * i + 2] * ri + a[3 * i + 2]);
    if (cxf) {
        const double *T = cxf + CXF_N * c;
        if (T[12] != 0.0) {
            double y[3];
            for (int j = 0; j < 3; j++) {
                y[j] = 0.0;
                y[j] += T[3 * j + 0] * x0;
                y[j] += T[3 * j + 1] * x1;
                y[j] += T[3 * j + 2] * x2;
            }
            x0 = y[0]; x1 = y[1]; x2 = y[2];
        }
        if (T[13] != 0.0) {
            x0 += T[9]; x1 += T[10]; x2 += T[11];
        }
    }
    return make_double4(x0, x1, x2, 0.0);
}

// facet normal and area: facnrm (src/shape/facnrm.c:13-25), cross
// (src/util/cross.c), normalize (src/util/normalize.c)
__device__ inline double4 facet_normal(double4 p0, double4 p1, double4 p2, double *area)
{
    double a0 = p1.x - p0.x, a1 = p1.y - p0.y, a2 = p1.z - p0.z;
    double b0 = p2.x - p1.x, b1 = p2.y - p1.y, b2 = p2.z - p1.z;
    double c0 = a1 * b2 - a2 * b1;
    double c1 = a2 * b0 - a0 * b2;
    double c2 = a0 * b1 - a1 * b0;
    if (area) *area = 0.5 * sqrt(c0 * c0 + c1 * c1 + c2 * c2);
    double norm = 0.0;
    norm += c0 * c0;
    norm += c1 * c1;
    norm += c2 * c2;
    norm = sqrt(norm);
    if (norm != 0.0) {
        c0 /= norm; c1 /= norm; c2 /= norm;
    }
    return make_double4(c0, c1, c2, 0.0);
}

// Vertices and facets in one launch: threads [0, nf) realize a facet from
// its three corners, which they compute themselves with the vertex formula
// (same operations, so the same bits as the vertex threads), and threads
// [nf, nf + nv) realize the vertices for the later stages.
template <typename P>
__device__ inline void realize_vf(int k, int nv, int nf, const double *__restrict__ a, const double *__restrict__ u,
                                  const P &par, const int *__restrict__ vcomp, const double *__restrict__ cxf,
                                  const int *__restrict__ fv, double4 *__restrict__ vx, double4 *__restrict__ fn,
                                  double *__restrict__ area, int4 *__restrict__ fvi)
{
    if (k < nf) {
        int i0 = fv[3 * k + 0], i1 = fv[3 * k + 1], i2 = fv[3 * k + 2];
        fvi[k] = make_int4(i0, i1, i2, 0);
        fn[k] = facet_normal(realize_vertex(i0, a, u, par, vcomp, cxf), realize_vertex(i1, a, u, par, vcomp, cxf),
                             realize_vertex(i2, a, u, par, vcomp, cxf), &area[k]);
    } else if (k < nf + nv) {
        vx[k - nf] = realize_vertex(k - nf, a, u, par, vcomp, cxf);
    }
}
__global__ void k_realize_vf(int nv, int nf, const double *__restrict__ a, const double *__restrict__ u,
                             const double *__restrict__ r, const double *__restrict__ scale,
                             const int *__restrict__ vcomp, const double *__restrict__ cxf,
                             const int *__restrict__ fv, double4 *__restrict__ vx, double4 *__restrict__ fn,
                             double *__restrict__ area, int4 *__restrict__ fvi)
{
    realize_vf(blockIdx.x * blockDim.x + threadIdx.x, nv, nf, a, u, ArrayParams{r, scale}, vcomp, cxf, fv, vx, fn, area,
               fvi);
}

// vertex normal = normalized sum of attached facet normals, in af order
// (src/shape/realize_mod.c:550-563)
__device__ inline void store_vnormal(int i, double n0, double n1, double n2, double4 *__restrict__ vn,
                                     float4 *__restrict__ vnf)
{
    double norm = 0.0;
    norm += n0 * n0;
    norm += n1 * n1;
    norm += n2 * n2;
    norm = sqrt(norm);
    if (norm != 0.0) {
        n0 /= norm; n1 /= norm; n2 /= norm;
    }
    vn[i] = make_double4(n0, n1, n2, 0.0);
    if (vnf) vnf[i] = make_float4((float)n0, (float)n1, (float)n2, 0.0f);
}
__device__ inline void realize_vnormal(int i, const int *__restrict__ af_ptr, const int *__restrict__ af_idx,
                                       const double4 *__restrict__ fn, double4 *__restrict__ vn,
                                       float4 *__restrict__ vnf)
{
    double n0 = 0.0, n1 = 0.0, n2 = 0.0;
    for (int j = af_ptr[i]; j < af_ptr[i + 1]; j++) {
        double4 fnj = fn[af_idx[j]];
        n0 += fnj.x; n1 += fnj.y; n2 += fnj.z;
    }
    store_vnormal(i, n0, n1, n2, vn, vnf);
}
__global__ void k_realize_vnormals(int nv, const int *__restrict__ af_ptr, const int *__restrict__ af_idx,
                                   const double4 *__restrict__ fn, double4 *__restrict__ vn,
                                   float4 *__restrict__ vnf)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nv) realize_vnormal(i, af_ptr, af_idx, fn, vn, vnf);
}

// ------------------------------------------------------------- transforms

// Vertex coordinates in each view's frame: cotrans(v, oa, x, 1) then
// += orbit_offset (src/shape/posvis.c:159-166; 0.0 for the engine's views).
__device__ inline double4 view_vertex(const FrameGeom &g, double4 x)
{
    double t[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        t[r] = 0.0;
        t[r] += g.oa[3 * r + 0] * x.x;
        t[r] += g.oa[3 * r + 1] * x.y;
        t[r] += g.oa[3 * r + 2] * x.z;
        t[r] += g.off[r];
    }
    return make_double4(t[0], t[1], t[2], 0.0);
}
template <typename T4>
__global__ void k_xform(const FrameGeom *__restrict__ geoms, const double4 *__restrict__ vx, int nv,
                        T4 *__restrict__ vt)
{
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const FrameGeom &g = geoms[blockIdx.y];
    vt[g.vt_base + i] = view_vertex(g, vx[i]);
}

// -------------------------------------------------------------- binning

// Resident 256-thread blocks per SM the binning kernel's registers must
// allow: it waits on dependent loads (normal and corners, then the bin
// atomics), so more blocks in flight hide more of that latency.
#ifndef BIN_MIN_BLOCKS
#define BIN_MIN_BLOCKS 6
#endif

// Facet culling, bounding box, outbnd flag and POSrect bookkeeping of
// posvis (src/shape/posvis.c:142-199, 322-364), then one bin entry per
// overlapped 16x16 tile. Bin order is arbitrary; the raster needs none.
__device__ inline bool faces_viewer(const FrameGeom &g, const double4 &nb)
{
    double nz = 0.0;
    nz += g.oa[6] * nb.x;
    nz += g.oa[7] * nb.y;
    nz += g.oa[8] * nb.z;
    return nz > 0.0;
}
// A facet that faces the viewer, its corners in the view's frame: its entries.
__device__ inline void bin_facet(int f, const FrameGeom &g, const double4 p0, const double4 p1, const double4 p2,
                                 FrameState &st, int *__restrict__ bin_count, int2 *__restrict__ bin_ids, int cap)
{
    const double kmpp = g.kmpp;
    const int n = g.n;
    double xmin = dmin_((double)p0.x, dmin_((double)p1.x, (double)p2.x));
    double xmax = dmax_((double)p0.x, dmax_((double)p1.x, (double)p2.x));
    double ymin = dmin_((double)p0.y, dmin_((double)p1.y, (double)p2.y));
    double ymax = dmax_((double)p0.y, dmax_((double)p1.y, (double)p2.y));
    double imin_d = floor(xmin / kmpp - SMALLVAL + 0.5);
    double imax_d = floor(xmax / kmpp + SMALLVAL + 0.5);
    double jmin_d = floor(ymin / kmpp - SMALLVAL + 0.5);
    double jmax_d = floor(ymax / kmpp + SMALLVAL + 0.5);
    int imin = clamp_lo(imin_d), imax = clamp_hi(imax_d);
    int jmin = clamp_lo(jmin_d), jmax = clamp_hi(jmax_d);
    if (imin < -n || imax > n || jmin < -n || jmax > n)
        st.outbnd = 1;
    int i1 = max(imin, -n), i2 = min(imax, n), j1 = max(jmin, -n), j2 = min(jmax, n);
    if (i1 > n || i2 < -n || j1 > n || j2 < -n) {
        atomicMin(&st.ofr_i[0], max(imin, -n));
        atomicMax(&st.ofr_i[1], min(imax, n));
        atomicMin(&st.ofr_j[0], max(jmin, -n));
        atomicMax(&st.ofr_j[1], min(jmax, n));
        atomicMin(&st.ofr_ov[0], dkey(imin_d));
        atomicMax(&st.ofr_ov[1], dkey(imax_d));
        atomicMin(&st.ofr_ov[2], dkey(jmin_d));
        atomicMax(&st.ofr_ov[3], dkey(jmax_d));
        return;
    }
    int tx0 = (i1 + n) / TILE_W, tx1 = (i2 + n) / TILE_W;
    int ty0 = (j1 + n) / TILE_W, ty1 = (j2 + n) / TILE_W;
    {
        // facets inside one tile (most of them): lanes of a warp with the
        // same tile reserve their slots with one atomic
        const unsigned act = __activemask();
        const bool single = (tx0 == tx1) && (ty0 == ty1);
        const unsigned sm = __ballot_sync(act, single);
        if (single) {
            const int tile = g.tile_base + tx0 * g.tiles_x + ty0;
            const int lane = threadIdx.x & 31;
            const unsigned peers = __match_any_sync(sm, tile);
            const int leader = __ffs(peers) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(&bin_count[tile], __popc(peers));
            base = __shfl_sync(peers, base, leader);
            const int slot = base + __popc(peers & ((1u << lane) - 1u));
            if (slot < cap) {
                int ti0 = -n + tx0 * TILE_W, tj0 = -n + ty0 * TILE_W;
                int ri1 = max(i1, ti0) - ti0, ri2 = min(i2, ti0 + TILE_W - 1) - ti0;
                int rj1 = max(j1, tj0) - tj0, rj2 = min(j2, tj0 + TILE_W - 1) - tj0;
                bin_ids[(size_t)tile * cap + slot] = make_int2(f, ri1 | (ri2 << 4) | (rj1 << 8) | (rj2 << 12));
            } else {
                st.bin_overflow = 1;
            }
            return;
        }
    }
    for (int tx = tx0; tx <= tx1; tx++)
        for (int ty = ty0; ty <= ty1; ty++) {
            int tile = g.tile_base + tx * g.tiles_x + ty;
            int slot = atomicAdd(&bin_count[tile], 1);
            if (slot < cap) {
                // bbox clipped to the tile, relative to its corner, 4 bits per bound
                int ti0 = -n + tx * TILE_W, tj0 = -n + ty * TILE_W;
                int ri1 = max(i1, ti0) - ti0, ri2 = min(i2, ti0 + TILE_W - 1) - ti0;
                int rj1 = max(j1, tj0) - tj0, rj2 = min(j2, tj0 + TILE_W - 1) - tj0;
                bin_ids[(size_t)tile * cap + slot] = make_int2(f, ri1 | (ri2 << 4) | (rj1 << 8) | (rj2 << 12));
            } else {
                st.bin_overflow = 1;
            }
        }
}
template <typename T4>
__global__ void __launch_bounds__(256, BIN_MIN_BLOCKS) k_bin(const FrameGeom *__restrict__ geoms, int view0, int nf,
                      const int4 *__restrict__ fvi, const double4 *__restrict__ fn,
                      const T4 *__restrict__ vt, FrameState *__restrict__ states,
                      int *__restrict__ bin_count, int2 *__restrict__ bin_ids, int cap, VnormalArgs vna)
{
    grid_dep_trigger();
    grid_dep_wait();
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (vna.nv > 0 && blockIdx.y == gridDim.y - 1) {
        // a batched evaluation's last row of blocks: the vertex normals, which
        // like the binning wait for the facet normals only
        for (int i = f; i < vna.nv; i += gridDim.x * blockDim.x)
            realize_vnormal(i, vna.af_ptr, vna.af_idx, fn, vna.vn, vna.vnf);
        return;
    }
    if (f >= nf) return;
    int v = view0 + blockIdx.y;
    const FrameGeom &g = geoms[v];
    // the normal and the corner indices load together (the culling test
    // does not wait for the indices); the corners follow
    const double4 nb = fn[f];
    const int4 c = fvi[f];
    if (!faces_viewer(g, nb)) return;
    bin_facet(f, g, vt[g.vt_base + c.x], vt[g.vt_base + c.y], vt[g.vt_base + c.z], states[v], bin_count, bin_ids, cap);
}

__device__ inline FrameState blank_state()
{
    FrameState s;
    s.outbnd = 0;
    s.bin_overflow = 0;
    s.cov_i[0] = s.cov_j[0] = INT_MAX;
    s.cov_i[1] = s.cov_j[1] = INT_MIN;
    s.ofr_i[0] = s.ofr_j[0] = INT_MAX;
    s.ofr_i[1] = s.ofr_j[1] = INT_MIN;
    s.ofr_ov[0] = s.ofr_ov[2] = dkey(HUGENUMBER);
    s.ofr_ov[1] = s.ofr_ov[3] = dkey(-HUGENUMBER);
    s.idellim[0] = s.idoplim[0] = INT_MAX;
    s.idellim[1] = s.idoplim[1] = INT_MIN;
    s.dellim[0] = s.doplim[0] = dkey(HUGENUMBER);
    s.dellim[1] = s.doplim[1] = dkey(-HUGENUMBER);
    s.any_overflow = 0;
    return s;
}
__global__ void k_reset_state(FrameState *st, int nviews, int *bin_count, int ntiles)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nviews) st[i] = blank_state();
    for (int t = i; t < ntiles; t += gridDim.x * blockDim.x)
        bin_count[t] = 0;
}

// The first launch of a batched evaluation: everything that depends only on the
// parameters or on nothing, by ranges of blocks. The views' vertices
// (each realized on the fly with k_realize_vf's operations, then k_xform's),
// the facets' normals and areas, the vertices, the views' blank states and bin
// counts, and the cleared images. As separate launches on side branches (a
// reset kernel and three or four clears after one another) the clears ended
// 9.8 us after the parameters had arrived and binning started then; as one
// launch it starts after 2.8 (one frame). With few facets and views (bin_ids not
// null) the launch bins as well and sums the vertex normals, both from facets
// realized once more, and the evaluation has no binning launch: one frame of 2200
// facets 37.4 us on the device before, 31.0 so. It then bins into states and
// counts that the launch before it blanked, and blanks the other pair.
// Views whose vertices a thread writes, from the vertex realized once: as many
// as leave eight blocks of vertices per SM, at most 8. 1600 views of 4002
// vertices, evaluation on the device: 1731 us with a view per thread, 1713 with
// 4, 1711 with 8 and 1712 with 16 (the 205 MB of vertices take 32 us to write).
constexpr int FRONT_VIEWS = 8, FRONT_GRID = 148 * 8;
constexpr int VN_BLOCK = 32;               // vertices whose normals a block sums
struct FrontParams {
    const FrontArgs &a;
    __device__ double r(int i) const
    {
        double v = a.m.r[i];
        for (int k = 0; k < a.nchange; k++)
            if (a.change_at[k] == i) v = a.change_to[k];
        return v;
    }
    __device__ double scale(int k) const { return a.nscale ? a.scale[k] : a.m.scale[k]; }
};
__global__ void __launch_bounds__(256) k_front(const __grid_constant__ FrontArgs a)
{
    grid_dep_trigger();
    const ModelDev &m = a.m;
    const FrontParams par{a};
    __shared__ double4 normal[256];
    int b = blockIdx.x;
    if (b < a.nb_bin) {
        const int bpv = (m.nf + 255) / 256, v = b / bpv, f = (b - v * bpv) * 256 + threadIdx.x;
        if (f >= m.nf) return;
        const FrameGeom &g = a.geoms[v];
        const double4 x0 = realize_vertex(m.fv[3 * f], m.a, m.u, par, m.vcomp, m.cxf);
        const double4 x1 = realize_vertex(m.fv[3 * f + 1], m.a, m.u, par, m.vcomp, m.cxf);
        const double4 x2 = realize_vertex(m.fv[3 * f + 2], m.a, m.u, par, m.vcomp, m.cxf);
        if (!faces_viewer(g, facet_normal(x0, x1, x2, nullptr))) return;
        bin_facet(f, g, view_vertex(g, x0), view_vertex(g, x1), view_vertex(g, x2), a.states[v], a.bin_count, a.bin_ids,
                  a.cap);
        return;
    }
    b -= a.nb_bin;
    if (b < a.nb_vn) {
        // VN_BLOCK vertices' attached facets lie one after another in af_idx:
        // their normals by all threads (realized from the corners, as the
        // facets' own blocks run beside this one), the sums by a thread per
        // vertex
        const int i0 = b * VN_BLOCK, i = i0 + threadIdx.x;
        const int lo = m.af_ptr[i0], hi = m.af_ptr[min(i0 + VN_BLOCK, m.nv)];
        const bool sums = threadIdx.x < VN_BLOCK && i < m.nv;
        const int own0 = sums ? m.af_ptr[i] : 0, own1 = sums ? m.af_ptr[i + 1] : 0;
        double n0 = 0.0, n1 = 0.0, n2 = 0.0;
        for (int base = lo; base < hi; base += 256) {
            const int j = base + threadIdx.x;
            if (j < hi) {
                const int f = m.af_idx[j];
                normal[threadIdx.x] = facet_normal(realize_vertex(m.fv[3 * f], m.a, m.u, par, m.vcomp, m.cxf),
                                                   realize_vertex(m.fv[3 * f + 1], m.a, m.u, par, m.vcomp, m.cxf),
                                                   realize_vertex(m.fv[3 * f + 2], m.a, m.u, par, m.vcomp, m.cxf),
                                                   nullptr);
            }
            __syncthreads();
            for (int k = max(own0, base); k < min(own1, base + 256); k++) {
                const double4 nk = normal[k - base];
                n0 += nk.x; n1 += nk.y; n2 += nk.z;
            }
            __syncthreads();
        }
        if (sums) store_vnormal(i, n0, n1, n2, m.vn, m.vnf);
        return;
    }
    b -= a.nb_vn;
    if (b < a.nb_xform) {
        const int bpv = (m.nv + 255) / 256, v0 = b / bpv * a.views;
        const int i = (b % bpv) * 256 + threadIdx.x;
        if (i >= m.nv) return;
        const double4 x = realize_vertex(i, m.a, m.u, par, m.vcomp, m.cxf);
        for (int v = v0; v < min(v0 + a.views, a.nviews); v++) {
            const FrameGeom &g = a.geoms[v];
            a.vt[g.vt_base + i] = view_vertex(g, x);
        }
        return;
    }
    b -= a.nb_xform;
    if (b < a.nb_model) {
        realize_vf(b * 256 + threadIdx.x, m.nv, m.nf, m.a, m.u, par, m.vcomp, m.cxf, m.fv, m.vx, m.fn, m.area, m.fvi);
        return;
    }
    b -= a.nb_model;
    const int nb = gridDim.x - a.nb_bin - a.nb_vn - a.nb_xform - a.nb_model;
    const long long t0 = (long long)b * 256 + threadIdx.x, step = (long long)nb * 256;
    for (long long i = t0; i < a.nviews; i += step) a.blank[i] = blank_state();
    if (b == 0) {
        if (threadIdx.x < a.nscale) a.scale_out[threadIdx.x] = a.scale[threadIdx.x];
        if (threadIdx.x < a.nchange) a.r_out[a.change_at[threadIdx.x]] = a.change_to[threadIdx.x];
    }
    for (int k = 0; k < FrontArgs::CLEARS; k++) {
        // 16-byte stores, then the last bytes
        const size_t n16 = a.clear_bytes[k] / 16;
        int4 *p = reinterpret_cast<int4 *>(a.clear[k]);
        for (size_t i = (size_t)t0; i < n16; i += (size_t)step) p[i] = make_int4(0, 0, 0, 0);
        if (t0 < (long long)(a.clear_bytes[k] % 16)) a.clear[k][16 * n16 + t0] = 0;
    }
}

// ----------------------------------------------------------------- chi2

// Neumaier-compensated accumulator.
struct KSum {
    double s, c;
    __device__ void add(double x)
    {
        double t = s + x;
        if (fabs(s) >= fabs(x)) c += (s - t) + x; else c += (x - t) + s;
        s = t;
    }
    __device__ void merge(const KSum &o)
    {
        add(o.s);
        c += o.c;
    }
    __device__ double value() const { return s + c; }
};

__device__ inline KSum shfl_ksum(KSum a, int off)
{
    KSum b;
    b.s = __shfl_down_sync(0xffffffffu, a.s, off);
    b.c = __shfl_down_sync(0xffffffffu, a.c, off);
    return b;
}

// A frame's m2 and om from its items' partial sums (a compensated sum and its
// compensation each): lane l merges items l, l + 32, ..., then the lanes merge
// pairwise, a fixed order; read through L2 (other warps wrote them).
__device__ inline void frame_sums_warp(const double *part, int nitems, KSum &m2, KSum &om)
{
    const int lane = threadIdx.x & 31;
    m2 = om = KSum{0, 0};
    for (int k = lane; k < nitems; k += 32) {
        const double *p = part + 4 * k;
        const KSum a = {__ldcg(p), __ldcg(p + 1)}, b = {__ldcg(p + 2), __ldcg(p + 3)};
        m2.merge(a);
        om.merge(b);
    }
    for (int off = 16; off > 0; off >>= 1) {
        m2.merge(shfl_ksum(m2, off));
        om.merge(shfl_ksum(om, off));
    }
}

// Sum of obs^2 / var of each radar frame (src/shape/chi2.c:436-441), which
// depends on the data only: once per dataset, by the frame's chi-square items
// (each a share of its whole image), whose sums a warp per frame merges. A block
// per frame took 4.7 ms of finalize for one image of 2048 x 2048 bins.
__global__ void __launch_bounds__(256) k_item_o2(const int2 *items, const FrameHost *fh, const FrameGeom *geoms,
                                                 const double *obs, const double *oov, double *partials)
{
    __shared__ double red[8][2];
    const int2 item = items[blockIdx.x];
    if (item.y < 0) return;                    // the frame's geometry item
    const FrameHost &h = fh[item.x];
    const FrameGeom &g = geoms[h.view];
    const long long n = (long long)g.ndel * g.ndop, share = (n + h.nitems - 1) / h.nitems;
    const long long end = min(n, (item.y + 1) * share);
    KSum q = {0, 0};
    for (long long k = item.y * share + threadIdx.x; k < end; k += blockDim.x) {
        const double ob = obs[g.fit_base + k];
        q.add(ob * ob * oov[g.fit_base + k]);
    }
    for (int off = 16; off > 0; off >>= 1) q.merge(shfl_ksum(q, off));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { red[wid][0] = q.s; red[wid][1] = q.c; }
    __syncthreads();
    if (threadIdx.x != 0) return;
    q = {0, 0};
    for (int w = 0; w < 8; w++) q.merge(KSum{red[w][0], red[w][1]});
    double *part = partials + 4 * (size_t)blockIdx.x;
    part[0] = q.s; part[1] = q.c; part[2] = part[3] = 0.0;
}
__global__ void k_frame_o2(const FrameHost *fh, const double *partials, double *o2)
{
    KSum q, unused;
    frame_sums_warp(partials + 4 * (size_t)fh[blockIdx.x].item0, fh[blockIdx.x].nitems, q, unused);
    if (threadIdx.x != 0) return;
    o2[2 * blockIdx.x] = q.s;
    o2[2 * blockIdx.x + 1] = q.c;
}

// A frame's chi-square terms (src/shape/chi2.c:436-460).
__device__ void frame_chi2_from_sums(const FrameHost &h, const KSum &so2, const KSum &sm2, const KSum &som,
                                     shape_deldop_result &r)
{
    const double o2 = so2.value(), m2 = sm2.value(), om = som.value();
    double cal = h.cal_in;
    if (h.cal_floating)
        cal = (om > 0.0) ? om / m2 : SHAPE_TINYCALFACT;
    r.o2 = o2; r.m2 = m2; r.om = om; r.cal = cal;
    r.chi2 = h.weight * (o2 - 2 * cal * om + cal * cal * m2);
}

// A frame's posvis / pos2deldop outputs (limits, flags, log-factors), which
// do not depend on the chi-square sums.
__device__ void finalize_frame_geom(const FinalizeArgs &a, int fr, shape_deldop_result &r)
{
    const FrameHost &h = a.fh[fr];
    const FrameGeom &g = a.geoms[h.view];
    const FrameState &st = a.states[h.view];
    const double *ovf = (h.dop_index >= 0) ? a.ovf_out + (size_t)h.dop_index * DOP_OVF_TERMS : nullptr;
    const int n = g.n;
    r.xlim[0] = min(n, min(st.cov_i[0], st.ofr_i[0]));
    r.xlim[1] = max(-n, max(st.cov_i[1], st.ofr_i[1]));
    r.ylim[0] = min(n, min(st.cov_j[0], st.ofr_j[0]));
    r.ylim[1] = max(-n, max(st.cov_j[1], st.ofr_j[1]));
    r.outbnd = st.outbnd;
    r.posbnd_logfactor = 0.0;
    if (st.outbnd) {
        double oimin = dkey_inv(st.ofr_ov[0]), oimax = dkey_inv(st.ofr_ov[1]);
        double ojmin = dkey_inv(st.ofr_ov[2]), ojmax = dkey_inv(st.ofr_ov[3]);
        if (st.cov_i[0] != INT_MAX) {
            oimin = dmin_(oimin, (double)st.cov_i[0]);
            oimax = dmax_(oimax, (double)st.cov_i[1]);
            ojmin = dmin_(ojmin, (double)st.cov_j[0]);
            ojmax = dmax_(ojmax, (double)st.cov_j[1]);
        }
        double xfactor = (dmax_(oimax, n) - dmin_(oimin, -n) + 1) / (2 * n + 1);
        double yfactor = (dmax_(ojmax, n) - dmin_(ojmin, -n) + 1) / (2 * n + 1);
        r.posbnd_logfactor = log(xfactor * yfactor);
    }
    r.badradar = h.badradar;
    r.badradar_logfactor = h.badradar_logfactor;
    if (ovf && ovf[4] != 0.0) {       // model wider than the overflow spectrum
        r.badradar = 1;
        r.badradar_logfactor += ovf[5];
    }
    r.idellim[0] = min(g.ndel + 999999, st.idellim[0]);
    r.idellim[1] = max(-999999, st.idellim[1]);
    r.idoplim[0] = min(g.ndop + 999999, st.idoplim[0]);
    r.idoplim[1] = max(-999999, st.idoplim[1]);
    double dl0 = dmin_(HUGENUMBER, dkey_inv(st.dellim[0])), dl1 = dmax_(-HUGENUMBER, dkey_inv(st.dellim[1]));
    double pl0 = dmin_(HUGENUMBER, dkey_inv(st.doplim[0])), pl1 = dmax_(-HUGENUMBER, dkey_inv(st.doplim[1]));
    double dpp = a.set_delpp[h.set], fpp = a.set_doppp[h.set];
    r.dellim[0] = (dl0 - g.delshift) * dpp;
    r.dellim[1] = (dl1 - g.delshift) * dpp;
    r.doplim[0] = (pl0 - g.dopshift) * fpp - a.dop_extra[fr];
    r.doplim[1] = (pl1 - g.dopshift) * fpp + a.dop_extra[fr];
    if (g.dop1d) {                    // a spectrum has no delay axis
        r.idellim[0] = r.idellim[1] = 0;
        r.dellim[0] = r.dellim[1] = 0.0;
    }
}

// Overflow spectrum of a Doppler frame (src/shape/pos2doppler.c:451-499), by one
// warp: sums over the bins inside the frame's Doppler limits (count of nonzero
// bins, squares over the noise variance, cross section and its mean bin) and
// the flag of a model wider than the overflow spectrum.
__device__ void doppler_overflow_warp(const FinalizeArgs &a, const FrameHost &h)
{
    const int lane = threadIdx.x & 31;
    const FrameGeom &g = a.geoms[h.view];
    const FrameState &st = a.states[h.view];
    double *out = a.ovf_out + (size_t)h.dop_index * DOP_OVF_TERMS;
    if (!st.any_overflow) {
        if (lane < DOP_OVF_TERMS) out[lane] = 0.0;
        return;
    }
    const double *ov = a.ovf + g.ovf_base;
    const double variance = h.sdev * h.sdev;
    const int idop0 = g.idop0;
    const int j1 = max(st.idoplim[0] + idop0, 0), j2 = min(st.idoplim[1] + idop0, DOP_MAXOVERFLOW - 1);
    double o2 = 0.0, m2 = 0.0, xs = 0.0, dm = 0.0;
    for (int j = j1 + lane; j <= j2; j += 32) {
        const double v = ov[j];
        if (v != 0.0) {
            o2 += 1.0;
            m2 += v * v / variance;
            xs += v;
            dm += (j - idop0) * v;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        o2 += __shfl_down_sync(0xffffffffu, o2, o);
        m2 += __shfl_down_sync(0xffffffffu, m2, o);
        xs += __shfl_down_sync(0xffffffffu, xs, o);
        dm += __shfl_down_sync(0xffffffffu, dm, o);
    }
    if (lane != 0) return;
    if (xs != 0.0) dm /= xs;
    out[0] = o2; out[1] = m2; out[2] = xs; out[3] = dm;
    out[4] = out[5] = 0.0;
    const int lo = st.idoplim[0] + idop0, hi = st.idoplim[1] + idop0;
    if (lo < 0 || hi >= DOP_MAXOVERFLOW) {
        out[4] = 1.0;
        out[5] = log((max(hi, DOP_MAXOVERFLOW) - min(lo, 0)) / (1.0 * DOP_MAXOVERFLOW));
    }
}

// A radar frame's badradar term of the objective (src/shape/calc_fits.c:
// 545-550): dof * log-factor / views, summed over the views whose
// footprint was too wide; the flag when any of them was. One view: the
// frame's own result (which includes a Doppler frame's overflow term).
__device__ inline double frame_blog(const FrameHost &h, double frame_lf)
{
    return h.nviews > 1 ? h.dof * h.badradar_lfsum / h.nviews : h.dof * frame_lf / 1;
}
__device__ inline bool frame_bad(const FrameHost &h, int frame_bad)
{
    return frame_bad || (h.nviews > 1 && h.badradar_any);
}

// posbnd_logfactor of one POS view (src/shape/posvis.c:301-307).
__device__ double view_logfactor(const FrameGeom &g, const FrameState &st)
{
    const int n = g.n;
    double oimin = dkey_inv(st.ofr_ov[0]), oimax = dkey_inv(st.ofr_ov[1]);
    double ojmin = dkey_inv(st.ofr_ov[2]), ojmax = dkey_inv(st.ofr_ov[3]);
    if (st.cov_i[0] != INT_MAX) {
        oimin = dmin_(oimin, (double)st.cov_i[0]);
        oimax = dmax_(oimax, (double)st.cov_i[1]);
        ojmin = dmin_(ojmin, (double)st.cov_j[0]);
        ojmax = dmax_(ojmax, (double)st.cov_j[1]);
    }
    double xfactor = (dmax_(oimax, n) - dmin_(oimin, -n) + 1) / (2 * n + 1);
    double yfactor = (dmax_(ojmax, n) - dmin_(ojmin, -n) + 1) / (2 * n + 1);
    return log(xfactor * yfactor);
}


// ---- plane-of-sky frames (calc_poset, src/shape/calc_fits.c:1156-1330)

// The interpolation polynomial of cubic convolution with parameter -1 (the
// original kernel; resampim's CUBICPAR), in resampim's operations.
__device__ double cubicconv_w(double x)
{
    const double c = -1.0;
    const double ax = fabs(x);
    if (ax < 1) return (c + 2) * ax * ax * ax - (c + 3) * ax * ax + 1;
    if (ax < 2) return c * (ax * ax * ax - 5 * ax * ax + 8 * ax - 4);
    return 0.0;
}

// One sample of the resampling grid (src/util/resampim.c): the grid point
// of temporary column it and row jt, reached by resampim's running sums
// (x1start and y1start advance once per column, x1 and y1 once per row),
// read from the brightness image B ([-n..n]^2, j contiguous) by the
// frame's interpolation; 0 where the input pixels it needs leave the image.
__device__ double poset_sample(const double *B, int n, int side, int mode, double x1start, double y1start,
                               double dxx, double dyx, double dxy, double dyy, int it, int jt)
{
    double x1 = x1start, y1 = y1start;
    for (int k = 1; k < it; k++) { x1 += dxx; y1 += dyx; }
    for (int k = 1; k < jt; k++) { x1 += dxy; y1 += dyy; }
#define IM(i_, j_) B[(long long)((i_) + n) * side + ((j_) + n)]
    if (mode == SHAPE_RESAMPLE_NONE || mode == SHAPE_RESAMPLE_NEAREST) {
        const int ix = iround_(x1), iy = iround_(y1);
        return (ix >= -n && ix <= n && iy >= -n && iy <= n) ? IM(ix, iy) : 0.0;
    }
    const int ix = (int)floor(x1), iy = (int)floor(y1);
    if (mode == SHAPE_RESAMPLE_BILINEAR) {
        if (!(ix >= -n && ix < n && iy >= -n && iy < n)) return 0.0;
        const double t = x1 - ix, u = y1 - iy;
        return (1 - t) * (1 - u) * IM(ix, iy) + t * (1 - u) * IM(ix + 1, iy) + t * u * IM(ix + 1, iy + 1) +
               (1 - t) * u * IM(ix, iy + 1);
    }
    // cubic convolution: four interpolations along rows, then one along the column
    double v = 0.0;
    if (ix > -n && ix < n - 1 && iy > -n && iy < n - 1) {
        const double t = x1 - ix, u = y1 - iy;
        double xp[4];
        for (int k = -1; k <= 2; k++) xp[k + 1] = cubicconv_w(k - t);
        for (int l = -1; l <= 2; l++) {
            double xi = 0.0;
            for (int k = -1; k <= 2; k++) xi += xp[k + 1] * IM(ix + k, iy + l);
            v += cubicconv_w(l - u) * xi;
        }
    }
    return v;
#undef IM
}

// gridDim.x blocks per plane-of-sky frame (blockIdx.y), each a slice of its fit
// grid and of its sky pixels: the fit image by resampim (with rebinning when the grid undersamples the rendering by an integer factor
// and image_rebin is set; cubic convolution clipped at 0), checkposet's
// test of the lit pixels' corners against the rotated fit grid
// (src/util/checkposet.c), chi2_poset's sums with the floating
// calibration (src/shape/chi2.c) and the views' posbnd terms. The block that
// finishes a frame last merges the blocks' sums in block order. One block per
// frame left the chip idle: the stage of three frames of 181^2 pixels took
// 120 us, with 17 blocks a frame 27.
__global__ void __launch_bounds__(256) k_poset_frames(PosetArgs a)
{
    grid_dep_trigger();
    grid_dep_wait();
    __shared__ double red[5][32];
    __shared__ int redi[32];
    const PosetFrameDev F = a.frames[blockIdx.y];
    const LcPointDev &P = a.pts[F.point];
    const FrameGeom &go = a.geoms[P.obs_view], &gs = a.geoms[P.sun_view];
    const int n = go.n, side = go.side;
    const double *B = a.bimg + P.b_base;
    const int ncol = F.ncol, nrow = F.nrow;
    double *FIT = a.fit + F.img_base;
    const double *OBS = a.obs + F.img_base, *OOV = a.oov + F.img_base;
    // resampim's grid over the temporary image (1..xt2) x (1..yt2)
    int xb = 1, yb = 1;
    if (F.rebin) {
        xb = max(iround_(F.xwidth / (ncol - 1)), 1);
        yb = max(iround_(F.ywidth / (nrow - 1)), 1);
    }
    const int npix = xb * yb;
    const bool rebin = F.rebin && npix > 1;
    const int xt2 = rebin ? xb * ncol : ncol, yt2 = rebin ? yb * nrow : nrow;
    const double xstep = (F.mode == SHAPE_RESAMPLE_NONE) ? 1.0 : F.xwidth / (xt2 - 1);
    const double ystep = (F.mode == SHAPE_RESAMPLE_NONE) ? 1.0 : F.ywidth / (yt2 - 1);
    const double dxx = xstep * F.cosang, dxy = ystep * F.sinang;
    const double dyx = -xstep * F.sinang, dyy = ystep * F.cosang;
    const double x1s = F.x0 - ((xt2 - 1) / 2.0) * dxx - ((yt2 - 1) / 2.0) * dxy;
    const double y1s = F.y0 - ((xt2 - 1) / 2.0) * dyx - ((yt2 - 1) / 2.0) * dyy;
    double o2 = 0.0, m2 = 0.0, om = 0.0;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (int p = t0; p < ncol * nrow; p += step) {
        const int i = p / nrow + 1, j = p % nrow + 1;
        double v;
        if (rebin) {
            v = 0.0;
            for (int k = 1 + (i - 1) * xb; k < 1 + i * xb; k++)
                for (int l = 1 + (j - 1) * yb; l < 1 + j * yb; l++)
                    v += poset_sample(B, n, side, F.mode, x1s, y1s, dxx, dyx, dxy, dyy, k, l);
            v /= npix;
        } else {
            v = poset_sample(B, n, side, F.mode, x1s, y1s, dxx, dyx, dxy, dyy, i, j);
        }
        if (F.mode == SHAPE_RESAMPLE_CUBICCONV) v = fmax(0.0, v);
        FIT[p] = v;
        const double ob = OBS[p], w = OOV[p];
        o2 += ob * ob * w;
        m2 += v * v * w;
        om += v * ob * w;
    }
    // checkposet: every corner of a lit POS pixel against the fit grid
    const double xl1 = -F.xwidth / 2 - 0.5, xl2 = F.xwidth / 2 + 0.5;
    const double yl1 = -F.ywidth / 2 - 0.5, yl2 = F.ywidth / 2 + 0.5;
    double xmin = xl1, xmax = xl2, ymin = yl1, ymax = yl2;
    int bad = 0;
    const int cside = side + 1;
    for (int c = t0; c < cside * cside; c += step) {
        const int ci = c / cside - n, cj = c % cside - n;      // corner (ci, cj): ci, cj = -n..n+1
        bool lit = false;
        for (int di = -1; di <= 0 && !lit; di++)
            for (int dj = -1; dj <= 0 && !lit; dj++) {
                const int pi = ci + di, pj = cj + dj;
                if (pi >= -n && pi <= n && pj >= -n && pj <= n && B[(long long)(pi + n) * side + (pj + n)] > 0.0)
                    lit = true;
            }
        if (!lit) continue;
        const double xs = (ci - 0.5) - F.x0, ys = (cj - 0.5) - F.y0;
        const double xf = xs * F.cosang + ys * F.sinang;
        const double yf = -xs * F.sinang + ys * F.cosang;
        if (xf < xl1) { bad = 1; xmin = fmin(xmin, xf); }
        else if (xf > xl2) { bad = 1; xmax = fmax(xmax, xf); }
        if (yf < yl1) { bad = 1; ymin = fmin(ymin, yf); }
        else if (yf > yl2) { bad = 1; ymax = fmax(ymax, yf); }
    }
    // block reductions: sums, extremes, the flag
    for (int off = 16; off > 0; off >>= 1) {
        o2 += __shfl_down_sync(0xffffffffu, o2, off);
        m2 += __shfl_down_sync(0xffffffffu, m2, off);
        om += __shfl_down_sync(0xffffffffu, om, off);
        xmin = fmin(xmin, __shfl_down_sync(0xffffffffu, xmin, off));
        xmax = fmax(xmax, __shfl_down_sync(0xffffffffu, xmax, off));
        ymin = fmin(ymin, __shfl_down_sync(0xffffffffu, ymin, off));
        ymax = fmax(ymax, __shfl_down_sync(0xffffffffu, ymax, off));
        bad |= __shfl_down_sync(0xffffffffu, bad, off);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __shared__ double ext[4][32];
    if (lane == 0) {
        red[0][wid] = o2; red[1][wid] = m2; red[2][wid] = om;
        ext[0][wid] = xmin; ext[1][wid] = xmax; ext[2][wid] = ymin; ext[3][wid] = ymax;
        redi[wid] = bad;
    }
    __syncthreads();
    double *part = a.part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * POSET_PART;
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        o2 = m2 = om = 0.0;
        for (int w = 0; w < nw; w++) {
            o2 += red[0][w]; m2 += red[1][w]; om += red[2][w];
            xmin = fmin(xmin, ext[0][w]); xmax = fmax(xmax, ext[1][w]);
            ymin = fmin(ymin, ext[2][w]); ymax = fmax(ymax, ext[3][w]);
            bad |= redi[w];
        }
        part[0] = o2; part[1] = m2; part[2] = om;
        part[3] = xmin; part[4] = xmax; part[5] = ymin; part[6] = ymax;
        part[7] = bad;
        __threadfence();                                      // the partials before the count
        s_last = (atomicAdd(&a.counters[blockIdx.y], 1) == (int)gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    o2 = m2 = om = 0.0;
    bad = 0;
    const double *all = a.part + (size_t)blockIdx.y * gridDim.x * POSET_PART;
#pragma unroll 4
    for (int b = 0; b < (int)gridDim.x; b++) {
        const double *q = all + (size_t)b * POSET_PART;
        o2 += __ldcg(q); m2 += __ldcg(q + 1); om += __ldcg(q + 2);
        xmin = fmin(xmin, __ldcg(q + 3)); xmax = fmax(xmax, __ldcg(q + 4));
        ymin = fmin(ymin, __ldcg(q + 5)); ymax = fmax(ymax, __ldcg(q + 6));
        bad |= __ldcg(q + 7) != 0.0;
    }
    shape_poset_result r;
    r.o2 = o2; r.m2 = m2; r.om = om;
    r.cal = (om > 0.0) ? om / m2 : SHAPE_TINYCALFACT;
    r.chi2 = F.weight * (o2 - 2 * r.cal * om + r.cal * r.cal * m2);
    r.badposet = bad;
    r.badposet_logfactor = bad ? log((xmax - xmin) * (ymax - ymin) / ((F.xwidth + 1) * (F.ywidth + 1))) : 0.0;
    const FrameState &so = a.states[P.obs_view], &ss = a.states[P.sun_view];
    r.outbnd = (so.outbnd ? 1 : 0) | (ss.outbnd ? 2 : 0);
    r.posbnd_logsum = 0.0;
    if (so.outbnd) r.posbnd_logsum += 0.5 * F.dof * view_logfactor(go, so);
    if (ss.outbnd) r.posbnd_logsum += 0.5 * F.dof * view_logfactor(gs, ss);
    a.res[blockIdx.y] = r;
}

// Natural cubic spline second derivatives and evaluation (the role of
// spline/splint in src/shape/calc_fits.c:1923-1933). The tridiagonal system
//   h[i-1] y2[i-1] + 2 (h[i-1] + h[i]) y2[i] + h[i] y2[i+1]
//     = 6 ((y[i+1]-y[i])/h[i] - (y[i]-y[i-1])/h[i-1]),   y2[0] = y2[n-1] = 0,
// is solved with each row divided by its span x[i+1] - x[i-1] (lower
// coefficient w = h[i-1]/span, diagonal 2, upper 1 - w): forward elimination
// keeps each row's multiplier of y2[i+1] in y2[i] and its eliminated right-hand
// side, back substitution forms y2[i] = mult[i] y2[i+1] + r[i]. The reference
// solves the span-scaled rows in this order, so equal brightnesses give its fits
// to the bit (they are sums over tiles here, in another order than its). Multipliers and pivots depend on the epochs only and come from the
// host (spline_plan); what remains serial is r[i] = (rhs[i] - w r[i-1]) / piv
// and the back substitution. The quotient is Markstein's: q = RN(a RN(1/b)),
// then q + RN(1/b) (a - q b) with the residual exact in a fused multiply-add,
// which is RN(a / b); three dependent operations instead of a division's ten.
__device__ inline double div_by(double a, double b, double rb)
{
    const double q = a * rb;
    return fma(rb, fma(-q, b, a), q);
}

__device__ double splint_dev(const double *x, const double *y, const double *y2, int n, double t)
{
    int lo = 0, hi = n - 1;
    while (hi - lo > 1) {
        int mid = (lo + hi) / 2;
        if (x[mid] > t) hi = mid; else lo = mid;
    }
    double h = x[hi] - x[lo];
    double wl = (x[hi] - t) / h, wh = (t - x[lo]) / h;
    return wl * y[lo] + wh * y[hi] +
           ((wl * wl * wl - wl) * y2[lo] + (wh * wh * wh - wh) * y2[hi]) * (h * h) / 6.0;
}

// One block per lightcurve set: y from the tiles' brightness, spline to the
// observation epochs, chi2_lghtcrv (src/shape/chi2.c:1125-1170), posbnd sum
// (src/shape/calc_fits.c:1651-1679, 1947).
//
// The recurrences (spline elimination and back substitution, the chi-square
// sums, the log-factor sum) stay serial in the reference's order, so equal
// brightnesses give its results to the bit; everything else, their operands included, is formed
// by the whole block first (in shared memory when a.smem_per_set > 0, else in
// the set's scratch). What bounds it is their latency: with each step's slopes,
// pivot and division inside the recurrence, the finalize and summary stage of
// four sets of 200 points took 128 us; it takes 55.
__global__ void __launch_bounds__(1024) k_lc_finalize(LcFinalizeArgs a)
{
    grid_dep_trigger();
    grid_dep_wait();
    extern __shared__ double lsm[];
    const LcSetDev &S = a.sets[blockIdx.x];
    const int np = S.npts, n = S.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    // work arrays: y, y2, r, lower coefficients, pivots and their reciprocals
    // [np]; the chi-square terms [2 n]
    double *y = a.smem_per_set > 0 ? lsm : S.scratch, *y2 = y + np, *r = y2 + np, *ll = r + np, *pv = ll + np,
           *rpv = pv + np, *m2t = rpv + np, *omt = m2t + n;
    const double *w = S.spl, *piv = w + np, *rpiv = piv + np, *mult = rpiv + np, *span = mult + np;
    __shared__ int s_bnd;
    if (tid == 0) s_bnd = 0;
    __syncthreads();
    // a warp per point: its observer view's tiles in a fixed order
    for (int k = wid; k < np; k += nw) {
        const LcPointDev &P = a.pts[S.pt0 + k];
        const FrameGeom &go = a.geoms[P.obs_view];
        const double *part = a.tile_part + go.tile_base;
        const int nt = go.tiles_x * go.tiles_x;
        double sum = 0.0;
        for (int t = lane; t < nt; t += 32) sum += part[t];
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
        if (lane == 0) {
            sum = (sum == 0.0) ? 1.0e-40 : sum;
            y[k] = S.y[k] = sum;
            const FrameState &so = a.states[P.obs_view], &ss = a.states[P.sun_view];
            // a point's two posbnd terms are added one after the other
            double l0 = 0.0, l1 = 0.0;
            if (so.outbnd) { s_bnd = 1; l0 = 0.5 * view_logfactor(go, so); }
            if (ss.outbnd) { s_bnd = 1; l1 = 0.5 * view_logfactor(a.geoms[P.sun_view], ss); }
            ll[k] = l0;
            y2[k] = l1;
        }
    }
    __syncthreads();
    double lsum = 0.0;
    if (tid == 0 && s_bnd)
        for (int k = 0; k < np; k++) { lsum += ll[k]; lsum += y2[k]; }
    __syncthreads();
    for (int i = 1 + tid; i < np - 1; i += blockDim.x) {
        const double dslope = (y[i + 1] - y[i]) / (S.x[i + 1] - S.x[i]) - (y[i] - y[i - 1]) / (S.x[i] - S.x[i - 1]);
        r[i] = 6.0 * dslope / span[i];
        y2[i] = mult[i];
        ll[i] = w[i];
        pv[i] = piv[i];
        rpv[i] = rpiv[i];
    }
    __syncthreads();
    if (tid == 0) {
        double rp = 0.0;
        r[0] = 0.0;
#pragma unroll 4
        for (int i = 1; i < np - 1; i++) {
            rp = div_by(r[i] - ll[i] * rp, pv[i], rpv[i]);
            r[i] = rp;
        }
        double yn = 0.0;
        y2[np - 1] = 0.0;
#pragma unroll 4
        for (int i = np - 2; i > 0; i--) {
            yn = y2[i] * yn + r[i];
            y2[i] = yn;
        }
        y2[0] = 0.0;
    }
    __syncthreads();
    for (int k = tid; k < n; k += blockDim.x) {
        const double v = splint_dev(S.x, y, y2, np, S.t[k]) / 1;
        S.fit[k] = v;
        m2t[k] = v * v * S.oov[k];
        omt[k] = v * S.obs[k] * S.oov[k];
    }
    for (int k = tid; k < np; k += blockDim.x) S.y2[k] = y2[k];
    __syncthreads();
    if (tid == 0) {
        double m2 = 0.0, om = 0.0;
#pragma unroll 8
        for (int k = 0; k < n; k++) {
            m2 += m2t[k];
            om += omt[k];
        }
        const double o2 = S.o2;
        double cal = S.cal_in;
        if (S.cal_floating)
            cal = (om > 0.0) ? om / m2 : SHAPE_TINYCALFACT;
        double *o = a.set_out + 4 * blockIdx.x;
        o[0] = cal;
        o[1] = S.weight * (o2 - 2 * cal * om + cal * cal * m2);
        o[2] = s_bnd;
        o[3] = lsum;
    }
}

// Totals over all sets in dataset order: chi2 (src/shape/chi2.c:270-300),
// the posbnd / badradar flags and log-factors of calc_fits
// (src/shape/calc_fits.c:407-409, 511-550, 1947) and the objective's
// bad-model multipliers (src/shape/bestfit.c:806-866), no penalties.
//
// The totals are serial sums in dataset order (the reference's order). One
// warp: its lanes read 32 radar frames' results at a time (through L2, other
// warps of the launch may have written them), and every lane adds the values
// it is handed by shuffles, so the sums wait on no load.
__device__ void totals_warp(const SummaryArgs &a)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double chi2 = 0.0, chi2_dd = 0.0, chi2_lc = 0.0, chi2_ps = 0.0, plog = 0.0, blog = 0.0, pslog = 0.0;
    int posbnd = 0, badradar = 0, badposet = 0;
    for (int s = 0; s < a.nsets; s++) {
        const SetRec R = a.sets[s];
        double cs = 0.0;
        if (R.type == 2) {
            // plane-of-sky frames: chi2_poset's frame sum; calc_poset's
            // posbnd terms (dof/2 per view) and badposet terms (dof times
            // checkposet's log factor)
            for (int f = R.first; f < R.first + R.count; f++) {
                const shape_poset_result &r = a.ps_res[f];
                cs += r.chi2;
                if (r.outbnd) { posbnd = 1; plog += r.posbnd_logsum; }
                if (r.badposet) { badposet = 1; pslog += a.ps_frames[f].dof * r.badposet_logfactor; }
            }
            chi2_ps += cs;
        } else if (R.type == 0) {
            for (int f0 = 0; f0 < R.count; f0 += 32) {
                const int nb = min(32, R.count - f0), f = R.first + f0 + min(lane, nb - 1);
                const shape_deldop_result *r = a.results + f;
                const FrameHost &h = a.fh[f];
                const double c = __ldcg(&r->chi2);
                const bool out = lane < nb && __ldcg(&r->outbnd), bad = lane < nb && frame_bad(h, __ldcg(&r->badradar));
                const unsigned mo = __ballot_sync(full, out), mb = __ballot_sync(full, bad);
                double pl = 0.0, bl = 0.0;
                if (mo) pl = h.dof * __ldcg(&r->posbnd_logfactor);
                if (mb) bl = frame_blog(h, __ldcg(&r->badradar_logfactor));
#pragma unroll 8
                for (int k = 0; k < nb; k++) cs += __shfl_sync(full, c, k);
                for (unsigned m = mo; m; m &= m - 1) plog += __shfl_sync(full, pl, __ffs(m) - 1);
                for (unsigned m = mb; m; m &= m - 1) blog += __shfl_sync(full, bl, __ffs(m) - 1);
                posbnd |= mo != 0;
                badradar |= mb != 0;
            }
            chi2_dd += cs;
        } else {
            const double *o = a.lc_out + 4 * R.first;
            cs = o[1];
            if (o[2] != 0.0) posbnd = 1;
            plog += a.lc_dof[R.first] * (o[3] / a.lc_npts[R.first]);
            chi2_lc += cs;
        }
        chi2 += cs;
    }
    if (lane != 0) return;
    shape_eval_summary out;
    out.chi2 = chi2;
    out.dof = a.dof;
    out.chi2_deldop = chi2_dd;
    out.chi2_lghtcrv = chi2_lc;
    out.posbnd = posbnd;
    out.posbnd_logfactor = plog / a.dof;
    out.badradar = badradar;
    out.badradar_logfactor = blog / a.dof_radar;
    out.chi2_poset = chi2_ps;
    out.badposet = badposet;
    out.badposet_logfactor = badposet ? pslog / a.dof_poset : 0.0;
    double err = chi2 / a.dof;
    if (a.baddiam) err *= a.bad_objfactor * exp(a.baddiam_logfactor);
    if (posbnd) err *= a.bad_objfactor * exp(out.posbnd_logfactor);
    if (badposet) err *= a.bad_objfactor * exp(out.badposet_logfactor);
    if (badradar) err *= a.bad_objfactor * exp(out.badradar_logfactor);
    out.objective = err;
    out.penalties = 0.0;
    *a.out = out;
}

// The totals of an engine without radar frames.
__global__ void k_totals(SummaryArgs a)
{
    grid_dep_wait();
    totals_warp(a);
}

// One item's sums of m2 = fit^2/var and om = fit obs/var, left in m2 and om of
// thread 0 of the block with their compensations. The item is a share of
// the frame's lit box, the rows and columns that its footprints reach (the
// union over a smeared frame's views): outside it the fit is zero and adds
// nothing. Each thread adds U bins in plain FP64 and that sum with
// compensation to its own, then the threads' sums merge with compensation in a
// fixed order. A bin whose fit is zero adds exact zeros whatever its observation
// and variance are (an infinite 1/var included), inside the box as outside.
struct Chi2Frame {                             // a frame's constants
    int view, nviews, nitems, ndel, ndop, dop1d;
    long long base;
};
template <typename T>
__device__ void chi2_item(const Chi2Args &a, const Chi2Frame &h, const FrameState *states, int k, KSum &m2, KSum &om)
{
    constexpr int U = 4;                       // bins a thread keeps in flight
    const int tid = threadIdx.x, lane = tid & 31;
    __shared__ double red[CHI2_THREADS / 32][4];
    int r0 = INT_MAX, r1 = INT_MIN, c0 = INT_MAX, c1 = INT_MIN;
    for (int v = h.view - h.nviews + 1; v <= h.view; v++) {
        const FrameState &st = states[v];
        r0 = min(r0, st.idellim[0]); r1 = max(r1, st.idellim[1]);
        c0 = min(c0, st.idoplim[0]); c1 = max(c1, st.idoplim[1]);
    }
    r0 = max(r0, 1); r1 = min(r1, h.ndel); c0 = max(c0, 1); c1 = min(c1, h.ndop);
    const int C = c1 - c0 + 1;
    const int n = (r1 >= r0 && C > 0) ? (r1 - r0 + 1) * C : 0;
    const int share = (n + h.nitems - 1) / h.nitems;
    const int b0 = k * share, b1 = min(n, b0 + share);
    // a spectrum of the FP32 form is summed in FP64 and rounded once, here
    const bool spectrum = sizeof(T) == 4 && h.dop1d;
    m2 = om = KSum{0, 0};
    if (b0 + tid < b1) {
        int row = (b0 + tid) / C, col = (b0 + tid) - row * C;
        const int drow = CHI2_THREADS / C, dcol = CHI2_THREADS - drow * C;
        for (int b = b0 + tid; b < b1; b += CHI2_THREADS * U) {
            double f[U], ob[U], wv[U];
#pragma unroll
            for (int j = 0; j < U; j++) {
                const bool in = b + CHI2_THREADS * j < b1;
                const long long p = h.base + (long long)(r0 - 1 + row) * h.ndop + (c0 - 1 + col);
                f[j] = ob[j] = wv[j] = 0.0;
                if (in) {
                    if (spectrum) {
                        const float v = (float)a.fit64[p];
                        static_cast<float *>(a.fit)[p] = v;
                        f[j] = v;
                    } else {
                        f[j] = (double)static_cast<const T *>(a.fit)[p];
                    }
                    ob[j] = a.obs[p];
                    wv[j] = a.oov[p];
                }
                row += drow;
                col += dcol;
                if (col >= C) { col -= C; row++; }
            }
            double sm2 = 0.0, som = 0.0;
#pragma unroll
            for (int j = 0; j < U; j++) {
                if (f[j] == 0.0) continue;
                sm2 += f[j] * f[j] * wv[j];
                som += f[j] * ob[j] * wv[j];
            }
            m2.add(sm2);
            om.add(som);
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        m2.merge(shfl_ksum(m2, off));
        om.merge(shfl_ksum(om, off));
    }
    if (lane == 0) {
        double *r = red[tid >> 5];
        r[0] = m2.s; r[1] = m2.c; r[2] = om.s; r[3] = om.c;
    }
    __syncthreads();
    if (tid >= 32) return;
    const int w = lane & (CHI2_THREADS / 32 - 1);
    m2 = KSum{red[w][0], red[w][1]};
    om = KSum{red[w][2], red[w][3]};
    for (int off = CHI2_THREADS / 64; off > 0; off >>= 1) {
        m2.merge(shfl_ksum(m2, off));
        om.merge(shfl_ksum(om, off));
    }
}

// Chi-square partials, per-frame results and totals in one launch: a block per
// (frame, item). A frame's counter takes one count per item; the block that
// makes the frame's last count merges the frame's item partials and writes its
// chi-square terms (a block of its own has written the limits, flags and
// log-factors, and a Doppler frame's overflow terms), and the one that completes the last frame computes the totals in dataset order. Values another
// block wrote in this launch are read through L2 (__ldcg) after a fence.
// counters: [nframes] per frame, then the finished frames; zero before the
// launch.
//
// What bounds it is the chain of dependent loads, fences and counts, not the
// images: a warp per item of 512 bins of the whole image read 12.5 MB of 64
// frames for their 5 % of lit bins and counted 6100 times (stage 23 us); a block
// per share of the lit box (chi2_shares) counts 500 times (17 us).
template <typename T>
__global__ void __launch_bounds__(CHI2_THREADS) k_chi2_summary(Chi2Args ca, FinalizeArgs fa, SummaryArgs sa,
                                                               int *counters)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, it = blockIdx.x;
    // constant data: read before the wait
    const int2 item = ca.items[it];
    const int fr = item.x;
    const FrameHost &h = fa.fh[fr];
    const KSum o2pre = {ca.o2[2 * fr], ca.o2[2 * fr + 1]};
    const int nitems = h.nitems, item0 = h.item0;
    const FrameGeom &g = fa.geoms[h.view];
    const Chi2Frame cf = {h.view, h.nviews, nitems, g.ndel, g.ndop, g.dop1d, g.fit_base};
    grid_dep_wait();
    KSum m2 = {0, 0}, om = {0, 0};
    if (item.y < 0) {
        // the frame's geometry block
        if (threadIdx.x >= 32) return;
        if (h.dop_index >= 0) doppler_overflow_warp(fa, h);
        __syncwarp();
        if (lane == 0) finalize_frame_geom(fa, fr, fa.results[fr]);
    } else {
        chi2_item<T>(ca, cf, fa.states, item.y, m2, om);
        if (threadIdx.x >= 32) return;
    }
    int last = 0;
    if (lane == 0) {
        double *part = ca.partials + 4 * (size_t)it;
        part[0] = m2.s; part[1] = m2.c; part[2] = om.s; part[3] = om.c;
        __threadfence();                                      // the partials before the count
        last = (atomicAdd(&counters[fr], 1) == nitems);       // the shares and the geometry
    }
    last = __shfl_sync(full, last, 0);
    if (!last) return;                                        // warp-uniform
    __threadfence();
    frame_sums_warp(ca.partials + 4 * (size_t)item0, nitems, m2, om);
    int lastf = 0;
    if (lane == 0) {
        // a Doppler frame's sums start from its overflow spectrum's o2 and m2
        // (src/shape/chi2.c:745-747)
        KSum so2 = o2pre, sm2 = m2;
        if (h.dop_index >= 0) {
            const double *ovf = fa.ovf_out + (size_t)h.dop_index * DOP_OVF_TERMS;
            so2 = KSum{__ldcg(ovf), 0};
            so2.merge(o2pre);
            sm2 = KSum{__ldcg(ovf + 1), 0};
            sm2.merge(m2);
        }
        frame_chi2_from_sums(h, so2, sm2, om, fa.results[fr]);
        __threadfence();                                      // the results before the count
        lastf = fa.nframes == 1 || atomicAdd(&counters[fa.nframes], 1) == fa.nframes - 1;
    }
    lastf = __shfl_sync(full, lastf, 0);
    if (!lastf) return;
    __threadfence();
    totals_warp(sa);
}

}  // namespace

// ------------------------------------------------------------- launchers

void launch_realize_vf(const ModelDev &m, cudaStream_t s)
{
    const int B = 256;
    k_realize_vf<<<(m.nf + m.nv + B - 1) / B, B, 0, s>>>(m.nv, m.nf, m.a, m.u, m.r, m.scale, m.vcomp, m.cxf, m.fv,
                                                          m.vx, m.fn, m.area, m.fvi);
}

void launch_realize_vn(const ModelDev &m, cudaStream_t s)
{
    const int B = 256;
    k_realize_vnormals<<<(m.nv + B - 1) / B, B, 0, s>>>(m.nv, m.af_ptr, m.af_idx, m.fn, m.vn,
                                                          m.vnf);
}

void launch_realize(const ModelDev &m, cudaStream_t s)
{
    launch_realize_vf(m, s);
    launch_realize_vn(m, s);
}

void launch_reset_state(FrameState *st, int nviews, int *bin_count, int ntiles, cudaStream_t s)
{
    int n = nviews > ntiles ? nviews : ntiles;
    int blocks = (n + 255) / 256;
    if (blocks > 4 * 148) blocks = 4 * 148;
    if (blocks < (nviews + 255) / 256) blocks = (nviews + 255) / 256;
    k_reset_state<<<blocks, 256, 0, s>>>(st, nviews, bin_count, ntiles);
}

void launch_front(const FrontArgs &a0, cudaStream_t s)
{
    FrontArgs a = a0;
    const long long bpv = (a.m.nv + 255) / 256;
    a.views = (int)std::min<long long>(FRONT_VIEWS, std::max<long long>(1, bpv * a.nviews / FRONT_GRID));
    a.nb_xform = (int)(bpv * ((a.nviews + a.views - 1) / a.views));
    a.nb_model = (a.m.nf + a.m.nv + 255) / 256;
    size_t words = (size_t)a.nviews;
    for (size_t n : a.clear_bytes) words = n / 16 > words ? n / 16 : words;
    // four 16-byte stores a thread, at most four blocks per SM
    size_t nb = (words + 1023) / 1024;
    nb = nb < 1 ? 1 : nb > 4 * 148 ? 4 * 148 : nb;
    a.nb_bin = a.bin_ids ? a.nviews * ((a.m.nf + 255) / 256) : 0;
    a.nb_vn = a.bin_ids ? (a.m.nv + VN_BLOCK - 1) / VN_BLOCK : 0;
    k_front<<<a.nb_bin + a.nb_vn + a.nb_xform + a.nb_model + (int)nb, 256, 0, s>>>(a);
}

void launch_xform_f64(const FrameGeom *g, int nviews, const double4 *vx, int nv, double4 *vt, cudaStream_t s,
                      bool pdl)
{
    dim3 grid((nv + 255) / 256, nviews);
    launch_k(k_xform<double4>, grid, dim3(256), 0, s, pdl, g, vx, nv, vt);
}


void launch_bin_f64(const FrameGeom *g, int view0, int nviews, const ModelDev &m, const double4 *vt,
                    FrameState *st, int *bin_count, int2 *bin_ids, int cap, cudaStream_t s, bool pdl, bool vnormals)
{
    // the vertex normals' blocks are one more row of the grid; where the views
    // take all that a grid may have (65535), a launch of their own
    if (vnormals && nviews + 1 > 65535) {
        launch_realize_vn(m, s);
        vnormals = false;
    }
    dim3 grid((m.nf + 255) / 256, nviews + (vnormals ? 1 : 0));
    const VnormalArgs vna = {vnormals ? m.nv : 0, m.af_ptr, m.af_idx, m.vn, m.vnf};
    launch_k(k_bin<double4>, grid, dim3(256), 0, s, pdl, g, view0, m.nf, (const int4 *)m.fvi, (const double4 *)m.fn,
             vt, st, bin_count, bin_ids, cap, vna);
}


void launch_frame_o2(const int2 *items, int nitems, const FrameHost *fh, int nframes, const FrameGeom *geoms,
                     const double *obs, const double *oov, double *partials, double *o2, cudaStream_t s)
{
    if (nframes <= 0) return;
    k_item_o2<<<nitems, 256, 0, s>>>(items, fh, geoms, obs, oov, partials);
    k_frame_o2<<<nframes, 32, 0, s>>>(fh, partials, o2);
}

void launch_poset_frames(const PosetArgs &a, cudaStream_t s, bool pdl)
{
    if (a.nframes <= 0) return;
    launch_k(k_poset_frames, dim3(a.blocks, a.nframes), dim3(256), 0, s, pdl, a);
}

// Shared memory one set needs (0 when it exceeds the block's budget: the
// kernel then works on the global arrays).
size_t lc_finalize_words(int npts, int n) { return 6 * (size_t)npts + 2 * (size_t)n; }
size_t lc_finalize_smem(int npts, int n)
{
    size_t b = sizeof(double) * lc_finalize_words(npts, n);
    return b <= LC_FINALIZE_SMEM_MAX ? b : 0;
}

cudaError_t configure_lc_finalize()
{
    return cudaFuncSetAttribute(k_lc_finalize, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)LC_FINALIZE_SMEM_MAX);
}

void launch_lc_finalize(const LcFinalizeArgs &a, cudaStream_t s, bool pdl)
{
    if (a.nsets <= 0) return;
    launch_k(k_lc_finalize, dim3(a.nsets), dim3(1024), a.smem_per_set, s, pdl, a);
}

void launch_chi2_summary(const Chi2Args &ca, const FinalizeArgs &fa, const SummaryArgs &sa, int *counters,
                         int fp32, cudaStream_t s, bool pdl)
{
    const int blocks = ca.nitems;                    // one block per item
    if (blocks <= 0) return;
    if (fp32) launch_k(k_chi2_summary<float>, dim3(blocks), dim3(CHI2_THREADS), 0, s, pdl, ca, fa, sa, counters);
    else launch_k(k_chi2_summary<double>, dim3(blocks), dim3(CHI2_THREADS), 0, s, pdl, ca, fa, sa, counters);
}

void launch_totals(const SummaryArgs &a, cudaStream_t s, bool pdl)
{
    launch_k(k_totals, dim3(1), dim3(32), 0, s, pdl, a);
}

}  // namespace shape
