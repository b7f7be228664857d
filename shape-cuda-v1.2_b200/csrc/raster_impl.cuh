// Tile rasterizer with fused delay-Doppler synthesis (T: the synthesis type,
// double in raster_f64.cu, compiled without FMA contraction, or float in
// raster_f32.cu).
//
// One CTA owns one 16x16 tile of one POS view. Coverage and depth are posvis's
// own FP64 expressions in both forms (src/shape/posvis.c:205-292), evaluated
// facet by facet rather than pixel by pixel:
//
//   A  each thread takes a facet of the tile's bin (filled by k_bin, in any
//      order), bounds the pixels it can cover row by row by its edges (FP32,
//      conservative) and leaves the facet with those pixels in shared memory;
//   B  each pixel tests its candidates with the exact expressions and shades
//      its winner;
//   C  in radar views each lit pixel adds its delay-Doppler footprint
//      (src/shape/pos2deldop.c:305-535) to the frame's fit image, so POS maps
//      never travel through HBM unless they are asked for.
//
// posvis walks the facets in index order and a facet takes a pixel when
// z > zz, so its final winner is the largest depth, the lowest index among
// equals: no order is needed for it, and no sort. Only cos(e) of a limb pixel,
// whose winner's smoothed normal faces away, depends on the order (it stays
// that of the last earlier winner whose normal faced the viewer); such a
// pixel steps back through its earlier winners (pixel_history).
//
// What bounds it: instruction issue and latency, not memory (the tile's data
// come from L2). A facet of a 20000-pixel body spans about 4 pixels: the exact
// test runs once per (facet, covered pixel) instead of once per pixel of every
// facet that meets a warp's block, and nothing is sorted. Facets of hundreds of
// pixels are tested by all pixels instead (FEW); bodies of many layers go through
// the phases in chunks of facets (tile_chunks).
#pragma once

#include <algorithm>
#include <climits>
#include <cstddef>

#include "kernels.h"
#include "posmask_dev.cuh"

// Resident warps per SM that the register allocation must allow (radar views
// FP32 / FP64, sun and observer views), and the share of the SM's 256 KB that the CTAs' shared memory may
// take; the rest is L1, where the facets' vertices and the spills live. The
// kernels wait on those loads more than they issue, so both count. 128-thread
// CTAs, ms: 64 uneven frames in FP32 at 40 warps 0.106 with all of it shared
// and 0.105 with 80 %, at 32 warps 0.104, 0.099 with 80 % and 0.099 with 65;
// 16 frames of 511^2 0.222 and 0.214 at 40, 0.204 and 0.192 at 32. The sun and
// observer views hold less per tile (no synthesis; a sun view no shading
// either): 800 points' both launches 1.52 at 32 warps, 1.38 at 40 and 1.35 at
// 48, but 25 points' 0.067, 0.067 and 0.075 (48 leave them half a wave). One
// share for all of them: a launch that changes it waits until the SM is empty
// (25 points' evaluation 0.099 with one share, 0.107 with two).
#ifndef RASTER_WARPS_F32
#define RASTER_WARPS_F32 32
#endif
#ifndef RASTER_SHARED_PCT
#define RASTER_SHARED_PCT 80
#endif
#ifndef RASTER_WARPS_F64
#define RASTER_WARPS_F64 32
#endif
#ifndef RASTER_WARPS_MAPS
#define RASTER_WARPS_MAPS 40
#endif

namespace shape {

template <typename T> __device__ inline T tsin(T x);
template <> __device__ inline double tsin<double>(double x) { return sin(x); }
template <> __device__ inline float tsin<float>(float x) { return sinf(x); }
template <typename T> __device__ inline T tsinpi(T x);
template <> __device__ inline double tsinpi<double>(double x) { return sinpi(x); }
template <> __device__ inline float tsinpi<float>(float x) { return sinpif(x); }
template <typename T> __device__ inline T tpow(T x, T y);
template <> __device__ inline double tpow<double>(double x, double y) { return pow(x, y); }
template <> __device__ inline float tpow<float>(float x, float y) { return powf(x, y); }
template <typename T> __device__ inline T texp(T x);
template <> __device__ inline double texp<double>(double x) { return exp(x); }
template <> __device__ inline float texp<float>(float x) { return expf(x); }

// SINC2 / TRI / TRI2 macros (src/macros/func.h:6-8)
template <typename T> __device__ inline T sinc2(T x)
{
    T tmp = fabs((T)3.141592653589793 * x);
    if (tmp > (T)1.0e-4) {
        tmp = tsin<T>(tmp) / tmp;
        return tmp * tmp;
    }
    return (T)1.0;
}
template <typename T> __device__ inline T tri(T x) { T t = (T)1 - fabs(x); return t > (T)0 ? t : (T)0; }
template <typename T> __device__ inline T tri2(T x) { T t = (T)1 - fabs(x); return t > (T)0 ? t * t : (T)0; }

// radlaw for the facet-independent laws (src/shape/radlaw.c:44-148)
template <typename T> __device__ T radlaw_dev(const RadarLawDev &L, T c)
{
    T v = (T)-9.99, tan2inc, sin2inc, arg;
    switch (L.type) {
    case SHAPE_RADLAW_COSINE_DIFF:
        v = (T)L.diff_R * ((T)L.diff_C + 1) * (L.diff_linear ? c : tpow<T>(c, 2 * (T)L.diff_C - 1));
        break;
    case SHAPE_RADLAW_GAUSSIAN:
        if (c >= (T)L.qs_cos_cutoff) {
            tan2inc = 1 / (c * c) - 1;
            v = (T)L.qs_R * (T)L.qs_C * texp<T>(-(T)L.qs_C * tan2inc) / (c * c * c * c * c);
        } else v = 0;
        break;
    case SHAPE_RADLAW_HAGFORS:
        if (c >= (T)L.qs_cos_cutoff) {
            sin2inc = 1 - c * c;
            arg = c * c * c * c + (T)L.qs_C * sin2inc;
            v = (T)0.5 * (T)L.qs_R * (T)L.qs_C * tpow<T>(arg, (T)-1.5) / c;
        } else v = 0;
        break;
    case SHAPE_RADLAW_COSINE_QS:
        if (c >= (T)L.qs_cos_cutoff)
            v = (T)L.qs_R * ((T)L.qs_C + 1) * (L.qs_linear ? c : tpow<T>(c, 2 * (T)L.qs_C - 1));
        else v = 0;
        break;
    case SHAPE_RADLAW_GAUSSIAN_COSINE:
        v = (T)L.diff_R * ((T)L.diff_C + 1) * (L.diff_linear ? c : tpow<T>(c, 2 * (T)L.diff_C - 1));
        if (c >= (T)L.qs_cos_cutoff) {
            tan2inc = 1 / (c * c) - 1;
            v += (T)L.qs_R * (T)L.qs_C * texp<T>(-(T)L.qs_C * tan2inc) / (c * c * c * c * c);
        }
        break;
    case SHAPE_RADLAW_HAGFORS_COSINE:
        v = (T)L.diff_R * ((T)L.diff_C + 1) * (L.diff_linear ? c : tpow<T>(c, 2 * (T)L.diff_C - 1));
        if (c >= (T)L.qs_cos_cutoff) {
            sin2inc = 1 - c * c;
            arg = c * c * c * c + (T)L.qs_C * sin2inc;
            v += (T)0.5 * (T)L.qs_R * (T)L.qs_C * tpow<T>(arg, (T)-1.5) / c;
        }
        break;
    case SHAPE_RADLAW_COSINE_COSINE:
        v = (T)L.diff_R * ((T)L.diff_C + 1) * (L.diff_linear ? c : tpow<T>(c, 2 * (T)L.diff_C - 1));
        if (c >= (T)L.qs_cos_cutoff)
            v += (T)L.qs_R * ((T)L.qs_C + 1) * (L.qs_linear ? c : tpow<T>(c, 2 * (T)L.qs_C - 1));
        break;
    default:
        break;
    }
    return v;
}
// radlaw_dev out of line: the laws other than the plain cosine carry powers and
// exponentials.
template <typename T> __device__ __noinline__ T radlaw_call(const RadarLawDev &L, T c) { return radlaw_dev<T>(L, c); }

// pos2deldop constants of one frame in the raster's arithmetic type: the
// FP64 raster reads them from FrameGeom, the FP32 raster from the
// host-rounded float copies (FrameGeom::fdd), once per tile.
template <typename T>
struct DDC {
    T delfact, delshift, ax, ay, dopshift, const1, const2, one_over_spb;
    T xincr, yincr, dopdiff_bl, dopdiff_max, dopDC_vig, dopfftlen, kmpp, half_w;
    T spb_over_stride, stride, spb_sq, nsinc2_sq;
};

template <typename T> __device__ inline DDC<T> load_ddc(const FrameGeom &g);
template <> __device__ inline DDC<double> load_ddc<double>(const FrameGeom &g)
{
    DDC<double> c;
    c.delfact = g.delfact; c.delshift = g.delshift; c.ax = g.ax; c.ay = g.ay; c.dopshift = g.dopshift;
    c.const1 = g.const1; c.const2 = g.const2; c.one_over_spb = g.one_over_spb;
    c.xincr = g.xincr; c.yincr = g.yincr; c.dopdiff_bl = g.dopdiff_bl; c.dopdiff_max = g.dopdiff_max;
    c.dopDC_vig = g.dopDC_vig; c.dopfftlen = g.dopfftlen; c.kmpp = g.kmpp; c.half_w = g.sinc2width / 2.0;
    c.spb_over_stride = (double)g.spb_over_stride; c.stride = (double)g.stride;
    c.spb_sq = (double)g.spb_sq; c.nsinc2_sq = (double)g.nsinc2_sq;
    return c;
}
template <> __device__ inline DDC<float> load_ddc<float>(const FrameGeom &g)
{
    const float4 *p = reinterpret_cast<const float4 *>(g.fdd);
    const float4 a = p[0], b = p[1], d = p[2], e = p[3], f = p[4];
    DDC<float> c;
    c.delfact = a.x; c.delshift = a.y; c.ax = a.z; c.ay = a.w;
    c.dopshift = b.x; c.const1 = b.y; c.const2 = b.z; c.one_over_spb = b.w;
    c.xincr = d.x; c.yincr = d.y; c.dopdiff_bl = d.z; c.dopdiff_max = d.w;
    c.dopDC_vig = e.x; c.dopfftlen = e.y; c.kmpp = e.z; c.half_w = e.w;
    c.spb_over_stride = f.x; c.stride = f.y; c.spb_sq = f.z; c.nsinc2_sq = f.w;
    return c;
}

// FP64 delay and Doppler position of a lit pixel; a tile reduces them to the
// frame's limits (dd_bin_limits turns the extremes into bin limits).
struct PixPos {
    double del, dop;
};

// Delay / Doppler position and footprint of one lit POS pixel
// (src/shape/pos2deldop.c:318-367).
template <typename T>
struct PixDD {
    T delPOS, dopPOS, codefactor;
    T ddel0, dfrac;            // FP32 form: delPOS - idel_min, frac(dopPOS) from FP64
    int ifl;                   // FP32 form: floor(dopPOS) from FP64; column idop's offset is dfrac + (ifl - idop)
    int idel_min, idel_max, idop_min, idop_max;
    bool ok;   // in_bounds: the whole footprint lies inside the frame
};

__device__ inline PixDD<double> pixel_dd_setup(const FrameGeom &g, int x, int y, double z, PixPos &pp)
{
    using T = double;
    PixDD<T> d;
    d.delPOS = z * g.delfact + g.delshift;
    d.idel_min = __double2int_rd(d.delPOS - g.const1) + 1;
    d.idel_max = __double2int_ru(d.delPOS + g.const1) - 1;
    d.dopPOS = g.ax * (T)x + g.ay * (T)y + g.dopshift;
    const T half_w = g.sinc2width / 2.0;
    d.idop_min = __double2int_rd(d.dopPOS - g.dopdiff_max + 1 - half_w);
    d.idop_max = __double2int_rd(d.dopPOS + g.dopdiff_max + half_w);
    // a smeared frame's view adds 1/views of its cross-section (wscale; 1
    // for a frame of one view)
    d.codefactor = ((g.codemethod == SHAPE_CODE_SHORT)
                       ? sinc2<T>((d.dopPOS - g.dopDC_vig) / g.dopfftlen) : (T)1) * g.wscale;
    pp.del = (double)d.delPOS;
    pp.dop = (double)d.dopPOS;
    d.ok = (d.idel_min >= 1) && (d.idel_max <= g.ndel) && (d.idop_min >= 1) && (d.idop_max <= g.ndop) &&
           (d.idel_max - d.idel_min + 1 <= SHAPE_MAXBINS);
    return d;
}

// FP32 form: the pixel's delay and Doppler positions in FP64 from its FP64
// depth (src/shape/pos2deldop.c:318-367), so the bin range and the in-frame
// test are the FP64 form's, and the fractional offsets the FP32 response
// weights take are rounded from FP64 values.
__device__ inline PixDD<float> pixel_dd_setup_x(const FrameGeom &g, int x, int y, double z, PixPos &pp)
{
    PixDD<float> d;
    const double del = z * g.delfact + g.delshift;
    d.idel_min = __double2int_rd(del - g.const1) + 1;
    d.idel_max = __double2int_ru(del + g.const1) - 1;
    const double dop = g.ax * (double)x + g.ay * (double)y + g.dopshift;
    d.idop_min = __double2int_rd(dop - g.dopdiff_max + 1 - g.half_w);
    d.idop_max = __double2int_rd(dop + g.dopdiff_max + g.half_w);
    d.delPOS = (float)del;
    d.dopPOS = (float)dop;
    d.ddel0 = (float)(del - (double)d.idel_min);
    d.ifl = __double2int_rd(dop);
    d.dfrac = (float)(dop - (double)d.ifl);
    d.codefactor = g.fscale;
    if (g.codemethod == SHAPE_CODE_SHORT) d.codefactor *= sinc2<float>((float)((dop - g.dopDC_vig) / g.dopfftlen));
    pp.del = del;
    pp.dop = dop;
    d.ok = (d.idel_min >= 1) && (d.idel_max <= g.ndel) && (d.idop_min >= 1) && (d.idop_max <= g.ndop) &&
           (d.idel_max - d.idel_min + 1 <= SHAPE_MAXBINS);
    return d;
}

// Bin limits (idel_min, idel_max, idop_min, idop_max) of a set of lit
// pixels from the extremes of their FP64 delay and Doppler positions. Each
// bound is computed per pixel above by the same expression, a non-decreasing
// function of the position (floor/ceil of correctly rounded sums), so its
// extreme over the set is its value at the extreme position: the same
// integers as a min/max over the pixels' own bounds.
__device__ inline void dd_bin_limits(const FrameGeom &g, double dmin, double dmax, double pmin, double pmax, int *l)
{
    const double half_w = g.sinc2width / 2.0;
    l[0] = (int)floor(dmin - g.const1) + 1;
    l[1] = (int)ceil(dmax + g.const1) - 1;
    l[2] = (int)floor(pmin - g.dopdiff_max + 1 - half_w);
    l[3] = (int)floor(pmax + g.dopdiff_max + half_w);
}

// Delay response of image row idel for a pixel at delay bin delPOS
// (src/shape/pos2deldop.c:371-425).
//
// ddel = delPOS - idel. The fast path forms it as (delPOS - idel_min) - r
// with a literal r: both subtractions of integers are exact at these
// magnitudes, so the value is the same as delPOS - (idel_min + r).
template <typename T>
__device__ inline T del_resp(const FrameGeom &g, const DDC<T> &k, T delPOS, T ddel, int idel)
{
    const int spb = g.spb;
    T dc;
    if (g.codemethod != SHAPE_CODE_LONG_ORIG) {
        if (spb == 1) {
            dc = tri2<T>(ddel);
        } else if (spb == 2) {
            T arg = (delPOS - ((T)idel - k.const2)) / k.spb_over_stride;
            dc = tri<T>(arg) + tri<T>(arg - (T)0.5);
            dc *= dc / 4;
        } else {
            dc = 0;
            int m_min = max((int)floor((ddel - k.const2) * k.stride), 0);
            int m_max = min((int)ceil((ddel + k.const1) * k.stride), spb) - 1;
            T arg = (delPOS - ((T)idel - k.const2)) / k.spb_over_stride - (T)m_min * k.one_over_spb;
            for (int m = m_min; m <= m_max; m++) {
                dc += tri<T>(arg);
                arg -= k.one_over_spb;
            }
            dc *= dc / k.spb_sq;
        }
    } else {
        dc = tri2<T>(ddel / k.spb_over_stride);
    }
    return dc;
}

// Mean sinc^2 Doppler response of column idop over nsinc2^2 points
// (src/shape/pos2deldop.c:432-460); s2u = sin^2(pi * frac(dopPOS)) serves
// the nsinc2 == 1 case, where sin^2(pi*(dopPOS - idop)) = s2u.
// ddop = dopPOS - idop, formed like ddel above.
template <typename T>
__device__ inline T dop_resp(const FrameGeom &g, const DDC<T> &k, T dopPOS, T ddop, T s2u, int idop)
{
    const int nsinc2 = g.nsinc2;
    if (nsinc2 == 1) {
        const T t = fabs((T)3.141592653589793 * ddop);
        // FP32 form: the fast quotient (2 ulp; t*t is far from its
        // underflow range) in place of the IEEE division
        if constexpr (sizeof(T) == 4) return (t > 1.0e-4f) ? __fdividef(s2u, t * t) : 1.0f;
        else return (t > 1.0e-4) ? s2u / (t * t) : 1.0;
    }
    if (nsinc2 == 2) {
        T bl = dopPOS + k.dopdiff_bl - (T)idop;
        return (sinc2<T>(bl) + sinc2<T>(bl + k.xincr) + sinc2<T>(bl + k.yincr) +
                sinc2<T>(bl + k.xincr + k.yincr)) / 4;
    }
    T left = dopPOS + k.dopdiff_bl - (T)idop;
    T sm = 0;
    for (int i = 0; i < nsinc2; i++) {
        T arg = left;
        for (int j = 0; j < nsinc2; j++) {
            sm += sinc2<T>(arg);
            arg += k.xincr;
        }
        left += k.yincr;
    }
    return sm / k.nsinc2_sq;
}

// Footprint sizes of the register-resident path.
constexpr int FAST_ROWS = 2;
constexpr int FAST_COLS = 8;

// Delay and Doppler response of one pixel and its scatter into the frame's
// image (src/shape/pos2deldop.c:371-496): any code, sampling and footprint
// size. The common frames take pixel_dd_scatter_lean, so this stays out of
// line: its weight arrays would cost every pixel registers. A: the image's
// element type (the FP32 form adds Doppler spectra in FP64: every lit pixel of
// a spectrum lands in the same few hundred bins, so float sums would round
// thousands of times per bin).
template <typename T, typename A>
__device__ __noinline__ void pixel_dd_scatter(const RasterArgs &a, const FrameGeom &g, T cose, PixDD<T> d, A *dst)
{
    const DDC<T> k = load_ddc<T>(g);
    const T delPOS = d.delPOS, dopPOS = d.dopPOS;
    const int idel_min = d.idel_min, idel_max = d.idel_max, idop_min = d.idop_min, idop_max = d.idop_max;
    // FP32 form: the offsets from the FP64 positions (frac + integer)
    constexpr bool f32 = sizeof(T) == 4;
    T s2u = 0;
    if (g.nsinc2 == 1) {
        const T su = tsin<T>((T)3.141592653589793 * (f32 ? d.dfrac : (dopPOS - floor(dopPOS))));
        s2u = su * su;
    }
    auto ddop_of = [&](int idop) -> T { return f32 ? d.dfrac + (T)(d.ifl - idop) : dopPOS - (T)idop; };
    auto ddel_of = [&](int idel) -> T { return f32 ? d.ddel0 - (T)(idel - idel_min) : delPOS - (T)idel; };
    const T rl = radlaw_dev<T>(a.laws[g.law], cose) * k.kmpp * k.kmpp * d.codefactor;
    T del_c[SHAPE_MAXBINS];
    T dop_c[SHAPE_MAXBINS + 1];
    for (int idel = idel_min; idel <= idel_max; idel++)
        del_c[idel - idel_min] = del_resp<T>(g, k, delPOS, ddel_of(idel), idel);
    for (int idop = idop_min; idop <= idop_max; idop++)
        dop_c[min(idop - idop_min, SHAPE_MAXBINS)] = dop_resp<T>(g, k, dopPOS, ddop_of(idop), s2u, idop);
    T sdel = 0, sdop = 0;
    for (int idel = idel_min; idel <= idel_max; idel++) sdel += del_c[idel - idel_min];
    for (int idop = idop_min; idop <= idop_max; idop++) sdop += dop_c[min(idop - idop_min, SHAPE_MAXBINS)];
    // sum of del_c*dop_c over the footprint = (sum del_c) * (sum dop_c)
    // (src/shape/pos2deldop.c:462-466)
    const T amp = rl / (sdel * sdop);
    for (int idel = idel_min; idel <= idel_max; idel++) {
        T ad = amp * del_c[idel - idel_min];
        A *row = dst + (long long)(idel - 1) * g.ndop - 1;
        for (int idop = idop_min; idop <= idop_max; idop++)
            atomicAdd(row + idop, (A)(ad * dop_c[min(idop - idop_min, SHAPE_MAXBINS)]));
    }
}

// One footprint row of the FP32 form straight into the frame's fit image: the
// row's FAST_COLS-wide weights (zero beyond the footprint) are shifted by the
// misalignment m of the first bin (0..3 floats) into the 16-byte aligned groups
// that cover them and land as vector reductions; group lanes outside the
// footprint add zero, which leaves those cells unchanged. The shift is two
// rounds of conditional moves, so the lanes of a warp stay converged whatever
// their misalignments.
__device__ inline void red_row_f32(float4 *base, const float (&w)[FAST_COLS], float ad, int m, int nc)
{
    float v[12];
#pragma unroll
    for (int j = 0; j < 12; j++) v[j] = (j < FAST_COLS) ? w[j] : 0.0f;
    const bool s1 = (m & 1) != 0, s2 = (m & 2) != 0;
#pragma unroll
    for (int j = 11; j >= 0; j--) v[j] = s1 ? (j >= 1 ? v[j - 1] : 0.0f) : v[j];
#pragma unroll
    for (int j = 11; j >= 0; j--) v[j] = s2 ? (j >= 2 ? v[j - 2] : 0.0f) : v[j];
    atomicAdd(base, make_float4(ad * v[0], ad * v[1], ad * v[2], ad * v[3]));
    if (m + nc > 4) atomicAdd(base + 1, make_float4(ad * v[4], ad * v[5], ad * v[6], ad * v[7]));
    if (m + nc > 8) atomicAdd(base + 2, make_float4(ad * v[8], ad * v[9], ad * v[10], ad * v[11]));
}

// 1/x for x of ordinary size: the hardware's FP32 reciprocal, for FP64 refined
// by two Newton steps r += r (1 - x r), each of which doubles its 23 correct
// bits (the last step's rounding leaves at most an ulp).
__device__ inline float quick_rcp(float x) { return __fdividef(1.0f, x); }
__device__ inline double quick_rcp(double x)
{
    double r = (double)__fdividef(1.0f, (float)x);
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

// The common frames (FrameGeom::lean: delay response tri2 of the scaled offset,
// one sinc^2 point per pixel) with a footprint of at most FAST_ROWS x FAST_COLS
// bins. A column's Doppler response is sin^2(pi x)/(pi x)^2 with
// sin^2(pi x) = sin^2(pi frac) for every column, and only the responses' ratios
// to their sum count, so 1/x^2 stands for it: no sine, and no division but the
// reciprocals. A pixel within 1e-4/pi of a column's centre, where the reference
// takes 1 for that column (src/macros/func.h:6), goes the general way. False
// when it does.
template <typename T>
__device__ inline bool pixel_dd_scatter_lean(const RasterArgs &a, const FrameGeom &g, T cose, const PixDD<T> &d, T *fit)
{
    const int nr = d.idel_max - d.idel_min + 1, nc = d.idop_max - d.idop_min + 1;
    if (!g.lean || nr > FAST_ROWS || nc > FAST_COLS) return false;
    T frac;                                    // Doppler offset from the column at or below the pixel
    int i0;                                    // that column - idop_min
    if constexpr (sizeof(T) == 4) { frac = d.dfrac; i0 = d.ifl - d.idop_min; }
    else { const T fl = floor(d.dopPOS); frac = d.dopPOS - fl; i0 = (int)fl - d.idop_min; }
    const T near = (T)3.2e-5;                  // just above 1e-4 / pi
    if (frac < near || frac > (T)1 - near) return false;
    T dc[FAST_ROWS], pc[FAST_COLS];
    T sdel = 0, sdop = 0;
    const T sos = (T)g.lean_sos;
#pragma unroll
    for (int r = 0; r < FAST_ROWS; r++) {
        T dd;
        if constexpr (sizeof(T) == 4) dd = d.ddel0 - (T)r; else dd = d.delPOS - (T)(d.idel_min + r);
        dc[r] = (r < nr) ? tri2<T>(g.lean_sos == 1 ? dd : dd / sos) : (T)0;
        sdel += dc[r];
    }
#pragma unroll
    for (int c = 0; c < FAST_COLS; c++) {
        const T x = frac + (T)(i0 - c);        // exact to a T's rounding of its own size
        pc[c] = (c < nc) ? quick_rcp(x * x) : (T)0;
        sdop += pc[c];
    }
    const T rl = (g.linlaw ? (sizeof(T) == 4 ? (T)g.famp : (T)g.amp) * cose
                           : radlaw_call<T>(a.laws[g.law], cose) * (T)g.kmpp * (T)g.kmpp) * d.codefactor;
    const T amp = rl / (sdel * sdop);
#pragma unroll
    for (int r = 0; r < FAST_ROWS; r++) {
        if (r >= nr) break;
        const T ad = amp * dc[r];
        T *cell = fit + (long long)(d.idel_min + r - 1) * g.ndop + (d.idop_min - 1);
        if constexpr (sizeof(T) == 4) {
            const int mis = (int)((reinterpret_cast<uintptr_t>(cell) >> 2) & 3);
            red_row_f32(reinterpret_cast<float4 *>(cell - mis), pc, ad, mis, nc);
        } else {
#pragma unroll
            for (int c = 0; c < FAST_COLS; c++)
                if (c < nc) atomicAdd(cell + c, ad * pc[c]);
        }
    }
    return true;
}

// ---- Frames with other responses, and Doppler spectra: footprints of at most
// STAGE_COLS columns with up to 3 x 3 sinc^2 points per pixel. A pixel's column
// weights are staged in shared memory (a row per lane of the warp; no local
// arrays) and added from there.
constexpr int STAGE_COLS = 11;             // odd: a warp's rows start in different banks
template <typename T> struct StageRow { T w[STAGE_COLS]; };

// Writes the pixel's Doppler weights (zero beyond the footprint) and returns
// the cross-section over the sum of all responses, so that a bin's
// contribution is the returned value x its delay response x its column's
// weight (src/shape/pos2deldop.c:432-496). Each of the NS x NS sinc^2 points of
// column k is sin^2(pi x)/(pi x)^2 at x = x0 - k, and sin^2(pi x) = sin^2(pi x0)
// for every column: NS^2 sines per pixel instead of NS^2 per column.
template <typename T, int NS>
__device__ inline T stage_columns(const FrameGeom &g, const PixDD<T> &d, T *w)
{
    T frac;
    int i0;
    if constexpr (sizeof(T) == 4) { frac = d.dfrac; i0 = d.ifl - d.idop_min; }
    else { const T fl = floor(d.dopPOS); frac = d.dopPOS - fl; i0 = (int)fl - d.idop_min; }
    const int nc = d.idop_max - d.idop_min + 1;
    T x0[NS * NS], s2[NS * NS];
#pragma unroll
    for (int i = 0; i < NS; i++)
#pragma unroll
        for (int j = 0; j < NS; j++) {
            const T x = frac + (NS > 1 ? (T)(g.dopdiff_bl + i * g.yincr + j * g.xincr) : (T)0);
            const T sn = tsinpi<T>(x - rint(x));
            x0[i * NS + j] = x;
            s2[i * NS + j] = sn * sn * (T)0.10132118364233778;        // 1 / pi^2
        }
    T sum = 0;
    for (int c = 0; c < STAGE_COLS; c++) {
        T v = 0;
        if (c < nc) {
#pragma unroll
            for (int k = 0; k < NS * NS; k++) {
                const T x = x0[k] + (T)(i0 - c);
                const T r2 = quick_rcp(x * x);
                // the reference's |pi x| > 1e-4
                v += (fabs((T)3.141592653589793 * x) > (T)1.0e-4) ? s2[k] * r2 : (T)1;
            }
            if (NS > 1) v = v / (NS * NS);
            sum += v;
        }
        w[c] = v;
    }
    return sum;
}
template <typename T>
__device__ __noinline__ T stage_pixel(const RasterArgs &a, const FrameGeom &g, T cose, PixDD<T> d, T *w)
{
    const T sdop = g.nsinc2 == 1 ? stage_columns<T, 1>(g, d, w)
                 : g.nsinc2 == 2 ? stage_columns<T, 2>(g, d, w) : stage_columns<T, 3>(g, d, w);
    T sdel = 1;                            // a spectrum's delay response
    if (!g.dop1d) {
        const DDC<T> k = load_ddc<T>(g);
        sdel = 0;
        for (int e = d.idel_min; e <= d.idel_max; e++)
            sdel += del_resp<T>(g, k, d.delPOS, sizeof(T) == 4 ? d.ddel0 - (T)(e - d.idel_min) : d.delPOS - (T)e, e);
    }
    return radlaw_call<T>(a.laws[g.law], cose) * (T)g.kmpp * (T)g.kmpp * d.codefactor / (sdel * sdop);
}
// Whether stage_pixel serves the frame and the footprint.
template <typename T>
__device__ inline bool stage_fits(const FrameGeom &g, const PixDD<T> &d)
{
    return g.nsinc2 <= 3 && d.idop_max - d.idop_min < STAGE_COLS;
}
// The rows of a staged delay-Doppler footprint, added to the frame's image.
template <typename T>
__device__ __noinline__ void scatter_staged(const FrameGeom &g, PixDD<T> d, T amp, const T *w, T *fit)
{
    const DDC<T> k = load_ddc<T>(g);
    const int nc = d.idop_max - d.idop_min + 1;
    for (int e = d.idel_min; e <= d.idel_max; e++) {
        const T ad = amp * del_resp<T>(g, k, d.delPOS, sizeof(T) == 4 ? d.ddel0 - (T)(e - d.idel_min) : d.delPOS - (T)e, e);
        if (ad == (T)0) continue;
        T *cell = fit + (long long)(e - 1) * g.ndop + (d.idop_min - 1);
        if constexpr (sizeof(T) == 4) {
            // aligned 16-byte reductions; lanes outside the footprint add zero
            const int mis = (int)((reinterpret_cast<uintptr_t>(cell) >> 2) & 3);
            float4 *grp = reinterpret_cast<float4 *>(cell - mis);
            for (int c = -mis; c < nc; c += 4, grp++) {
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = (c + j >= 0 && c + j < nc) ? ad * w[c + j] : 0.0f;
                atomicAdd(grp, make_float4(v[0], v[1], v[2], v[3]));
            }
        } else {
            for (int c = 0; c < nc; c++) atomicAdd(cell + c, ad * w[c]);
        }
    }
}
// The staged spectra of a warp's pixels (mask: the lanes that have one; o1, amp:
// each lane's first column and factor), added to the frame's spectrum: lane l
// sums column cb + l over the warp's pixels in FP64 and adds it once, where one
// atomic per pixel and column met on the few hundred bins that all of a
// spectrum's pixels share. All lanes of the warp call it together.
template <typename T, typename A>
__device__ inline void add_spectra(unsigned mask, int o1, T amp, int c1, int c2, const StageRow<T> *rows, A *spec)
{
    const int lane = threadIdx.x & 31;
    for (int cb = c1; cb <= c2; cb += 32) {
        const int c = cb + lane;
        double sum = 0.0;
        for (unsigned m = mask; m; m &= m - 1) {
            const int p = __ffs(m) - 1;
            const int k = c - __shfl_sync(0xffffffffu, o1, p);
            const T ap = __shfl_sync(0xffffffffu, amp, p);
            if (k >= 0 && k < STAGE_COLS) sum += (double)(ap * rows[p].w[k]);
        }
        if (c <= c2 && sum != 0.0) atomicAdd(spec + (c - 1), (A)sum);
    }
}

// A Doppler pixel whose footprint leaves the spectrum adds its contributions
// to the frame's overflow spectrum instead (src/shape/pos2doppler.c:399-414):
// the same weights as pixel_dd_scatter's generic path (one row, delay
// response 1), bins clipped to the overflow spectrum.
template <typename T>
__device__ __noinline__ void pixel_dop_overflow(const RasterArgs &a, const FrameGeom &g, T cose, PixDD<T> d)
{
    const DDC<T> k = load_ddc<T>(g);
    const int idop_min = d.idop_min, idop_max = d.idop_max;
    T s2u = 0;
    if (g.nsinc2 == 1) {
        T fr;
        if constexpr (sizeof(T) == 4) fr = d.dfrac; else fr = d.dopPOS - floor(d.dopPOS);
        const T su = tsin<T>((T)3.141592653589793 * fr);
        s2u = su * su;
    }
    const T rl = radlaw_dev<T>(a.laws[g.law], cose) * k.kmpp * k.kmpp * d.codefactor;
    T dop_c[SHAPE_MAXBINS + 1];
    for (int idop = idop_min; idop <= idop_max; idop++) {
        T ddop;
        if constexpr (sizeof(T) == 4) ddop = d.dfrac + (T)(d.ifl - idop); else ddop = d.dopPOS - (T)idop;
        dop_c[min(idop - idop_min, SHAPE_MAXBINS)] = dop_resp<T>(g, k, d.dopPOS, ddop, s2u, idop);
    }
    T sdop = 0;
    for (int idop = idop_min; idop <= idop_max; idop++) sdop += dop_c[min(idop - idop_min, SHAPE_MAXBINS)];
    const T amp = rl / ((T)1 * sdop);
    double *ov = a.ovf + g.ovf_base;
    const int idop1 = max(idop_min, -g.idop0), idop2 = min(idop_max, -g.idop0 + DOP_MAXOVERFLOW - 1);
    for (int idop = idop1; idop <= idop2; idop++)
        atomicAdd(ov + idop + g.idop0, (double)(amp * (T)1 * dop_c[min(idop - idop_min, SHAPE_MAXBINS)]));
}
// Warp-wide extremes with the hardware warp reduction (one instruction per
// 32-bit word); 64-bit order-preserving keys (dkey) reduce their high words
// first, then the low words of the lanes holding the extreme high word.
__device__ inline int warp_min(int v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ inline int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ inline unsigned long long warp_kmin(unsigned long long k)
{
    const unsigned hi = __reduce_min_sync(0xffffffffu, (unsigned)(k >> 32));
    const unsigned lo = __reduce_min_sync(0xffffffffu, ((unsigned)(k >> 32) == hi) ? (unsigned)k : 0xffffffffu);
    return ((unsigned long long)hi << 32) | lo;
}
__device__ inline unsigned long long warp_kmax(unsigned long long k)
{
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, ((unsigned)(k >> 32) == hi) ? (unsigned)k : 0u);
    return ((unsigned long long)hi << 32) | lo;
}
// Candidate facets a pixel holds, and those a tile holds beyond them. A convex
// body has one layer of facets (a few pixels on shared edges two), a 3 % rough
// 32768-facet body up to 14 at its limb; a tile with more is rastered in chunks
// (tile_chunks).
constexpr int CAND = 8;
constexpr int CAND_MORE = 512;

// A pixel's winner: facet (-1: none), depth, s and t, and the facet and (s, t)
// that cos(e) comes from (gf < 0: none).
struct PixelHit {
    int f, gf;
    double z, s, t, gs, gt;
};

// A facet's edges over a tile (facet_edges): t, s - t and 1 - s as linear functions
// c0 + cx li + cy lj of the pixel, raised by what they may be off, and the rows
// (bits 0-15) and columns (16-31) of its box.
struct FacetEdges {
    float c0[3], cx[3], cy[3];
    unsigned box;
};
// A bin of few entries, most of many pixels: a coarse model in a large window. A
// thread per facet that lists its pixels takes them one after the other while
// its CTA waits, so in the kernels for such views (RasterArgs::few) phase A keeps
// a bin's edges and boxes if it has at most FEW entries, and in phase B each
// pixel tests all of them. Device time of an evaluation with lists and so, us,
// FP32: one frame of 1001^2 pixels, 8000 facets, 142 and 109; 16 of 301^2, 128
// facets, 123 and 98; 25 lightcurve points of up to 257^2, 512 facets, 110 and 78;
// 4 frames of 511^2, 8192 facets, 131 and 118. With more entries the lists are as
// fast (one frame of 801^2, 32768 facets, some 25 a tile: 146 with lists, 138
// with FEW 24, 145 with 32).
constexpr int FEW = 24;

// Shared memory of a tile's CTA of NT threads. The exact terms of the bin's
// facets are kept when the bin has at most NT of them (most tiles); otherwise a
// pixel forms those of its own facets again.
template <typename T, int NT>
struct TileShared {
    union {
        struct {
            double term[10][NT];                     // FacetTerms of bin entry k in column k
            union {
                unsigned short cand[TILE_PIX][CAND]; // bin entries that may cover the pixel
                FacetEdges edge[FEW];                // a bin of at most FEW entries: theirs
            };
        };
        PixelHit hit[TILE_PIX];                      // tile_chunks: the outcome
        StageRow<T> stage[NT];                       // phase C: a row per thread
    };
    double xs[TILE_W], ys[TILE_W];         // pixel centres
    int cnt[TILE_PIX];                     // candidates (may exceed CAND)
    union {
        unsigned more[CAND_MORE];          // further ones: entry | pixel << 16
        struct {
            unsigned more_chunk[CAND_MORE / 2];  // tile_chunks: the same
            int2 fl[NT];                         // ... and the chunk's bin entries
        };
    };
    unsigned long long lim[4];             // the frame's delay and Doppler extremes so far
    int cov[4];                            // ... and covered-pixel bbox
    int n;                                 // entries of more (may exceed CAND_MORE)
    int m;                                 // tile_chunks: facets of a scanned chunk so far
};

// The terms of posvis's s, t, z expressions for one facet
// (src/shape/posvis.c:210-228), rounded operation by operation so that no
// multiply-add is fused in either translation unit.
struct FacetTerms {
    double x, y, z, A, B, C, D, E, F, den;
};
__device__ inline FacetTerms facet_terms(const double4 *vt, int4 c)
{
    const double4 p0 = vt[c.x], p1 = vt[c.y], p2 = vt[c.z];
    FacetTerms q;
    q.x = p0.x; q.y = p0.y; q.z = p0.z;
    q.A = __dsub_rn(p2.y, p1.y); q.B = __dsub_rn(p2.x, p1.x);
    q.C = __dsub_rn(p1.x, p0.x); q.D = __dsub_rn(p1.y, p0.y);
    q.E = __dsub_rn(p1.z, p0.z); q.F = __dsub_rn(p2.z, p1.z);
    q.den = __drcp_rn(__dsub_rn(__dmul_rn(q.C, q.A), __dmul_rn(q.B, q.D)));
    return q;
}
template <typename T, int NT>
__device__ inline void store_terms(TileShared<T, NT> &sh, int k, const FacetTerms &q)
{
    sh.term[0][k] = q.x; sh.term[1][k] = q.y; sh.term[2][k] = q.z; sh.term[3][k] = q.A; sh.term[4][k] = q.B;
    sh.term[5][k] = q.C; sh.term[6][k] = q.D; sh.term[7][k] = q.E; sh.term[8][k] = q.F; sh.term[9][k] = q.den;
}
template <typename T, int NT>
__device__ inline FacetTerms load_terms(const TileShared<T, NT> &sh, int k)
{
    return FacetTerms{sh.term[0][k], sh.term[1][k], sh.term[2][k], sh.term[3][k], sh.term[4][k],
                      sh.term[5][k], sh.term[6][k], sh.term[7][k], sh.term[8][k], sh.term[9][k]};
}
// s and t of the pixel centre (x0, y0); true where the facet covers it.
__device__ inline bool facet_st(const FacetTerms &q, double x0, double y0, double &s, double &t)
{
    const double dx = __dsub_rn(x0, q.x), dy = __dsub_rn(y0, q.y);
    s = __dmul_rn(__dsub_rn(__dmul_rn(dx, q.A), __dmul_rn(q.B, dy)), q.den);
    if (!((s >= -SHAPE_SMALLVAL) && (s <= 1.0 + SHAPE_SMALLVAL))) return false;
    t = __dmul_rn(__dsub_rn(__dmul_rn(q.C, dy), __dmul_rn(dx, q.D)), q.den);
    return (t >= -SHAPE_SMALLVAL) && (t <= __dadd_rn(s, SHAPE_SMALLVAL));
}
__device__ inline double facet_z(const FacetTerms &q, double s, double t)
{
    return __dadd_rn(__dadd_rn(q.z, __dmul_rn(s, q.E)), __dmul_rn(t, q.F));
}

// Component r of the observer-frame normal of facet f at (s, t) before its
// normalization: the interpolated vertex normals (smooth) or the facet normal,
// rotated (src/shape/posvis.c:146-148, 250-262), rounded op by op.
__device__ inline void body_normal64(const RasterArgs &a, int f, double s, double t, bool smooth, double m[3])
{
    if (smooth) {
        const int4 c = a.fvi[f];
        const double4 q0 = a.vn[c.x], q1 = a.vn[c.y], q2 = a.vn[c.z];
        m[0] = __dadd_rn(__dadd_rn(q0.x, __dmul_rn(s, __dsub_rn(q1.x, q0.x))), __dmul_rn(t, __dsub_rn(q2.x, q1.x)));
        m[1] = __dadd_rn(__dadd_rn(q0.y, __dmul_rn(s, __dsub_rn(q1.y, q0.y))), __dmul_rn(t, __dsub_rn(q2.y, q1.y)));
        m[2] = __dadd_rn(__dadd_rn(q0.z, __dmul_rn(s, __dsub_rn(q1.z, q0.z))), __dmul_rn(t, __dsub_rn(q2.z, q1.z)));
    } else {
        const double4 nb = a.fn[f];
        m[0] = nb.x; m[1] = nb.y; m[2] = nb.z;
    }
}
__device__ inline double view_row64(const FrameGeom &g, int r, const double m[3])
{
    return __dadd_rn(__dadd_rn(__dmul_rn(g.oa[3 * r], m[0]), __dmul_rn(g.oa[3 * r + 1], m[1])),
                     __dmul_rn(g.oa[3 * r + 2], m[2]));
}

// posvis's culling and bounding box of a facet for a tile whose bin overflowed (src/shape/posvis.c:146-199): the bin entry k_bin would
// have made, or false when the facet faces away or misses the tile.
__device__ inline bool facet_entry(const RasterArgs &a, const FrameGeom &g, const double4 *vt, int f, int ti0, int ti1,
                                   int tj0, int tj1, int2 &e)
{
    const double4 nb = a.fn[f];
    const double m[3] = {nb.x, nb.y, nb.z};
    if (!(view_row64(g, 2, m) > 0.0)) return false;
    const int4 c = a.fvi[f];
    const double4 p0 = vt[c.x], p1 = vt[c.y], p2 = vt[c.z];
    const double xmin = fmin(p0.x, fmin(p1.x, p2.x)), xmax = fmax(p0.x, fmax(p1.x, p2.x));
    const double ymin = fmin(p0.y, fmin(p1.y, p2.y)), ymax = fmax(p0.y, fmax(p1.y, p2.y));
    const double lo = (double)INT_MIN, hi = (double)INT_MAX;
    const int imin = (int)fmax(floor(__dadd_rn(__dsub_rn(__ddiv_rn(xmin, g.kmpp), SHAPE_SMALLVAL), 0.5)), lo);
    const int imax = (int)fmin(floor(__dadd_rn(__dadd_rn(__ddiv_rn(xmax, g.kmpp), SHAPE_SMALLVAL), 0.5)), hi);
    const int jmin = (int)fmax(floor(__dadd_rn(__dsub_rn(__ddiv_rn(ymin, g.kmpp), SHAPE_SMALLVAL), 0.5)), lo);
    const int jmax = (int)fmin(floor(__dadd_rn(__dadd_rn(__ddiv_rn(ymax, g.kmpp), SHAPE_SMALLVAL), 0.5)), hi);
    if (imin > ti1 || imax < ti0 || jmin > tj1 || jmax < tj0) return false;
    e = make_int2(f, (max(imin, ti0) - ti0) | ((min(imax, ti1) - ti0) << 4) | ((max(jmin, tj0) - tj0) << 8) |
                         ((min(jmax, tj1) - tj0) << 12));
    return true;
}

// The candidates of a pixel in turn: entry i (of candidates()) of pixel p, or -1
// where the overflow list's slot i - CAND holds another pixel's. few: a bin of at
// most FEW entries, the pixel's are the bits of sh.cnt; left: those to come.
template <typename T, int NT>
__device__ __forceinline__ int candidate(const TileShared<T, NT> &sh, bool few, int p, int i, unsigned &left)
{
    if (few) {
        const int k = __ffs(left) - 1;
        left &= left - 1;
        return k;
    }
    if (i < CAND) return sh.cand[p][i];
    const unsigned v = sh.more[i - CAND];
    return (int)(v >> 16) == p ? (int)(v & 0xffffu) : -1;
}
// How many to walk: the pixel's own, or all of the overflow list too.
template <typename T, int NT>
__device__ __forceinline__ int candidates(const TileShared<T, NT> &sh, bool few, int p)
{
    const int c = sh.cnt[p];
    if (few) return __popc(c);
    return c <= CAND ? c : CAND + sh.n;
}
// Whether bin entry k covers the pixel centre (x0, y0): its terms, s and t.
template <typename T, int NT>
__device__ inline bool entry_covers(const RasterArgs &a, const double4 *vt, const int2 *bin, const TileShared<T, NT> &sh,
                                    bool staged, int k, double x0, double y0, FacetTerms &q, double &s, double &t)
{
    q = staged ? load_terms<T, NT>(sh, k) : facet_terms(vt, a.fvi[bin[k].x]);
    return facet_st(q, x0, y0, s, t);
}

// cos(e)'s facet of a pixel whose final winner's smoothed normal faces away: the
// last of the pixel's earlier winners whose normal faces the viewer, by the sign
// of its view-z component (facet, s and t; facet -1 when there is none). Winners
// are the facets deeper than z0 (has: the pixel was not blank) and than every
// one of lower index, so the winner before facet f is the deepest facet below f:
// the walk steps back from the final winner. Forwards, through every winner from
// the first, 20 points of a 30 % rough body of 8192 facets took 348 us, 234
// backwards; 16 frames of 511^2 pixels of 32768 facets with 3 % roughness 257 and
// 240; 25 points of a smooth body the same.
template <typename T, int NT, bool FEW_VIEWS>
__device__ __noinline__ PixelHit pixel_history(const RasterArgs &a, const FrameGeom &g, const int2 *bin, int count,
                                               const TileShared<T, NT> &sh, int p, int below, bool has, double z0)
{
    const bool staged = count <= NT, few = FEW_VIEWS && count <= FEW;
    PixelHit h = {-1, -1, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double4 *vt = static_cast<const double4 *>(a.vt) + g.vt_base;
    const double x0 = sh.xs[p / TILE_W], y0 = sh.ys[p % TILE_W];
    const int nc = candidates<T, NT>(sh, few, p);
    for (;;) {
        unsigned left = sh.cnt[p];
        int bf = -1;
        double bz = 0.0, bs = 0.0, bt = 0.0;
        for (int i = 0; i < nc; i++) {
            const int k = candidate<T, NT>(sh, few, p, i, left);
            if (k < 0) continue;
            const int f = bin[k].x;
            if (f >= below) continue;
            FacetTerms q;
            double s, t;
            if (!entry_covers<T, NT>(a, vt, bin, sh, staged, k, x0, y0, q, s, t)) continue;
            const double z = facet_z(q, s, t);
            if (has && !(z > z0)) continue;
            if (bf < 0 || z > bz || (z == bz && f < bf)) { bf = f; bz = z; bs = s; bt = t; }
        }
        if (bf < 0) return h;
        double m[3];
        body_normal64(a, bf, bs, bt, true, m);
        if (view_row64(g, 2, m) > 0.0) {
            h.gf = bf; h.gs = bs; h.gt = bt;
            return h;
        }
        below = bf;
    }
}

// The edges of a facet of the tile whose first pixel centre is (x0, y0). In pixel
// units from the tile's corner, t, s - t and 1 - s are linear functions
// c0 + cx li + cy lj; a pixel the exact test accepts has them above -m, where m
// bounds the FP32 error of c0, cx and cy over the box and the exact test's own
// 1e-10. With u = 2^-24: A, den and kmpp rounded and multiplied give sx, sy, tx
// and ty to 5u, X and Y are right to 3u, so s0 and t0 are off by at most
// 10u mag (|X| + |Y|), their difference and the addition of m by 2u more, cx and
// cy by 6u, and the sum at a pixel of the box adds 2u of its terms and 7u 30 mag
// from cx and cy: in all 14u mag (|X| + |Y|) + 240u mag, 8.4e-7 and 1.5e-5 beside
// m's 2e-6 and 6.4e-5. Coefficients out of FP32's range, and a den below its normal
// numbers (facets of 1e19 length units), bound nothing (the whole box).
__device__ inline FacetEdges facet_edges(const FacetTerms &q, double x0, double y0, float ikm, double kmpp)
{
    const float den = (float)q.den, d = den * (float)kmpp;
    const float sx = (float)q.A * d, sy = -(float)q.B * d, tx = -(float)q.D * d, ty = (float)q.C * d;
    const float X = (float)(x0 - q.x) * ikm, Y = (float)(y0 - q.y) * ikm;
    const float mag = fabsf(sx) + fabsf(sy) + fabsf(tx) + fabsf(ty);
    const float m = 2e-6f * (1.0f + mag * (fabsf(X) + fabsf(Y) + 32.0f));
    const float s0 = sx * X + sy * Y, t0 = tx * X + ty * Y;
    FacetEdges e = {{t0 + m, s0 - t0 + m, 1.0f - s0 + m}, {tx, sx - tx, -sx}, {ty, sy - ty, -sy}, 0u};
    if (!(m < 1e24f) || fabsf(den) < 1.2e-38f)
        for (int k = 0; k < 3; k++) { e.c0[k] = 1.0f; e.cx[k] = e.cy[k] = 0.0f; }
    return e;
}

// Phase A for bin entry k: the pixels of each row of the facet's box that lie
// between its edges get the entry as a candidate. room: entries that sh.more
// takes.
template <typename T, int NT>
__device__ inline void bound_facet(int k, const FacetTerms &q, int box, double x0, double y0, float ikm, double kmpp,
                                   int room, TileShared<T, NT> &sh)
{
    const int ri1 = box & 15, ri2 = (box >> 4) & 15, rj1 = (box >> 8) & 15, rj2 = (box >> 12) & 15;
    const FacetEdges fe = facet_edges(q, x0, y0, ikm, kmpp);
    const float *c0 = fe.c0, *cx = fe.cx, *cy = fe.cy;
    float inv[3];
#pragma unroll
    for (int e = 0; e < 3; e++) inv[e] = -__fdividef(1.0f, fabsf(cy[e]));
    for (int ri = ri1; ri <= ri2; ri++) {
        float lo = (float)rj1, hi = (float)rj2;
#pragma unroll
        for (int e = 0; e < 3; e++) {
            // v + cy lj >= 0; cy = 0: v >= 0 bounds nothing (-inf, or NaN,
            // which fmaxf drops), v < 0 empties the row
            const float b = (c0[e] + cx[e] * (float)ri) * inv[e];
            lo = fmaxf(lo, cy[e] >= 0.0f ? b : lo);
            hi = fminf(hi, cy[e] >= 0.0f ? hi : -b);
        }
        const int ja = __float2int_ru(fminf(lo, 16.0f)), jb = __float2int_rd(fmaxf(hi, -1.0f));
        for (int j = ja; j <= jb; j++) {
            const int p = ri * TILE_W + j;
            const int i = atomicAdd(&sh.cnt[p], 1);
            if (i < CAND) {
                sh.cand[p][i] = (unsigned short)k;
            } else {
                const int o = atomicAdd(&sh.n, 1);
                if (o < room) sh.more[o] = (unsigned)k | ((unsigned)p << 16);
            }
        }
    }
}

// Phase A for entry k of a bin of at most FEW: its edges and box, for the pixels to
// test.
template <typename T, int NT>
__device__ inline void few_facet(int k, const FacetTerms &q, int box, double x0, double y0, float ikm, double kmpp,
                                 TileShared<T, NT> &sh)
{
    FacetEdges e = facet_edges(q, x0, y0, ikm, kmpp);
    // bits first .. last of a bound pair
    auto span = [](int first, int last) { return (2u << last) - (1u << first); };
    e.box = span(box & 15, (box >> 4) & 15) | span((box >> 8) & 15, (box >> 12) & 15) << 16;
    sh.edge[k] = e;
}
// The entries (bits) of such a bin that may cover the tile's pixel (li, lj).
template <typename T, int NT>
__device__ inline unsigned few_candidates(const TileShared<T, NT> &sh, int count, int li, int lj)
{
    const float fi = (float)li, fj = (float)lj;
    unsigned mask = 0;
    for (int k = 0; k < count; k++) {
        const FacetEdges &e = sh.edge[k];
        bool in = (e.box >> li & e.box >> (16 + lj) & 1u) != 0;
#pragma unroll
        for (int j = 0; j < 3; j++) in = in && e.c0[j] + e.cx[j] * fi + e.cy[j] * fj >= 0.0f;
        mask |= (unsigned)in << k;
    }
    return mask;
}

// A tile whose bin overflowed its capacity (then: all facets that meet the tile),
// or whose candidates overflow sh.more: phases A and B over chunks of at most NT
// facets, in any order, each pixel keeping the best so far (its thread's
// registers). A chunk whose own candidates overflow is tested facet by facet.
// The first pass over the chunks finds each pixel's winner. A pixel whose
// winner's smoothed normal faces away needs the last earlier winner that faces
// the viewer: winners are the facets deeper than every one of lower index, so
// the winner before facet f is the deepest facet below f, and each further pass
// steps back by one until the normal faces the viewer or none is left. The
// outcome goes to sh.hit.
//
// A pass per winner from the first one on, each pixel forming the facets' terms
// itself, took 5.3 ms for 8 views of 101^2 pixels of a 30 % rough body of 32768
// facets, 0.64 so; 8 views of a smooth one whose bins were too small 0.37 and
// 0.16.
template <typename T, int NT>
__device__ __noinline__ void tile_chunks(const RasterArgs &a, const FrameGeom &g, const int2 *bin, int count, int ti0,
                                         int ti1, int tj0, int tj1, bool smooth, TileShared<T, NT> &sh)
{
    constexpr int PP = TILE_PIX / NT, ROOM = CAND_MORE / 2;
    const int tid = threadIdx.x;
    const double4 *vt = static_cast<const double4 *>(a.vt) + g.vt_base;
    const double x0 = sh.xs[0], y0 = sh.ys[0];
    const float ikm = (float)g.ikm;
    const bool scan = count > a.cap;
    const int total = scan ? a.nf : count;
    PixelHit hit[PP];
    int below[PP];                             // facets a pass looks at (index below; 0: the pixel is done)
    double z0[PP];
    bool had[PP];
#pragma unroll
    for (int r = 0; r < PP; r++) {
        hit[r] = PixelHit{-1, -1, 0.0, 0.0, 0.0, 0.0, 0.0};
        below[r] = INT_MAX;
        // blank, or (accumulating calls) the depth the image already holds
        const int p = tid + r * NT, pi = ti0 + p / TILE_W, pj = tj0 + p % TILE_W;
        const long long q = g.pos_base + (long long)(pi + g.n) * g.side + (pj + g.n);
        had[r] = a.accumulate && pi <= ti1 && pj <= tj1 && a.pos_f[q] >= 0;
        z0[r] = had[r] ? static_cast<const double *>(a.pos_z)[q] : 0.0;
    }
    for (bool first = true;; first = false) {
        int bf[PP];
        double bz[PP], bs[PP], bt[PP];
#pragma unroll
        for (int r = 0; r < PP; r++) { bf[r] = -1; bz[r] = bs[r] = bt[r] = 0.0; }
        for (int next = 0;;) {
            // the next chunk
            int m = 0;
            __syncthreads();                   // the last one's lists are read
            for (int r = 0; r < PP; r++) sh.cnt[tid + r * NT] = 0;
            if (tid == 0) sh.n = sh.m = 0;
            if (!scan) {
                m = min(NT, total - next);
                if (tid < m) sh.fl[tid] = bin[next + tid];
                next += m;
            } else {
                while (next < total) {
                    int2 e;
                    const bool in = next + tid < total && facet_entry(a, g, vt, next + tid, ti0, ti1, tj0, tj1, e);
                    const int add = __syncthreads_count(in);
                    if (m + add > NT) break;   // they open the next chunk
                    if (in) sh.fl[atomicAdd(&sh.m, 1)] = e;
                    m += add;
                    next += NT;
                }
            }
            __syncthreads();
            if (m == 0) break;
            if (tid < m) {
                const int2 e = sh.fl[tid];
                const FacetTerms q = facet_terms(vt, a.fvi[e.x]);
                store_terms<T, NT>(sh, tid, q);
                bound_facet<T, NT>(tid, q, e.y, x0, y0, ikm, g.kmpp, ROOM, sh);
            }
            __syncthreads();
            const bool all = sh.n > ROOM;
#pragma unroll
            for (int r = 0; r < PP; r++) {
                if (below[r] == 0) continue;
                const int p = tid + r * NT, li = p / TILE_W, lj = p % TILE_W;
                unsigned none = 0;
                const int nc = all ? m : candidates<T, NT>(sh, false, p);
                for (int i = 0; i < nc; i++) {
                    const int k = all ? i : candidate<T, NT>(sh, false, p, i, none);
                    if (k < 0) continue;
                    const int2 e = sh.fl[k];
                    const int b = e.y;
                    if (all && (li < (b & 15) || li > ((b >> 4) & 15) || lj < ((b >> 8) & 15) || lj > ((b >> 12) & 15)))
                        continue;
                    if (e.x >= below[r]) continue;
                    const FacetTerms q = load_terms<T, NT>(sh, k);
                    double s, t;
                    if (!facet_st(q, sh.xs[li], sh.ys[lj], s, t)) continue;
                    const double z = facet_z(q, s, t);
                    if (had[r] && !(z > z0[r])) continue;
                    if (bf[r] < 0 || z > bz[r] || (z == bz[r] && e.x < bf[r])) {
                        bf[r] = e.x; bz[r] = z; bs[r] = s; bt[r] = t;
                    }
                }
            }
        }
        bool more = false;
#pragma unroll
        for (int r = 0; r < PP; r++) {
            if (below[r] == 0) continue;
            below[r] = 0;
            if (bf[r] < 0) continue;
            if (first) { hit[r].f = bf[r]; hit[r].z = bz[r]; hit[r].s = bs[r]; hit[r].t = bt[r]; }
            double m[3];
            body_normal64(a, bf[r], bs[r], bt[r], smooth, m);
            if (!smooth || view_row64(g, 2, m) > 0.0) {
                hit[r].gf = bf[r]; hit[r].gs = bs[r]; hit[r].gt = bt[r];
            } else {
                below[r] = bf[r];              // 0: no facet is below the first one
                more = more || bf[r] > 0;
            }
        }
        if (!__syncthreads_or(more)) break;
    }
    for (int r = 0; r < PP; r++) sh.hit[tid + r * NT] = hit[r];
    __syncthreads();
}

// apply_photo's brightness of a pixel lit at cos e = ce, cos i = ci
// (src/shape/apply_photo.c:85-133, 226-248).
__device__ inline double photo_brightness(const LcPointDev &P, double ce, double ci)
{
    if (P.law_type == SHAPE_OPTLAW_LAMBERT) return P.intensityfactor * P.scale * ci;
    if (P.law_type == SHAPE_OPTLAW_LOMMEL) return P.intensityfactor * P.scale * ci / (ci + ce);
    return P.intensityfactor * ci * (P.s_ls / (ci + ce) + P.s_l);
}

// posmask (src/shape/posmask.c:58-174): whether the point (pi, pj, z) of facet
// fac lies in shadow, by the sun view's depth and facet maps.
__device__ inline bool photo_shadowed(const RasterArgs &a, const FrameGeom &g, const LcPointDev &P, int pi, int pj,
                                      double z, int fac)
{
    const int n = g.n, side = g.side;
    const long long sun = a.geoms[P.sun_view].pos_base;
    const double *ZI = static_cast<const double *>(a.pos_z) + sun;
    const int *FI = a.pos_f + sun;
    const double xin[3] = {pi * g.kmpp, pj * g.kmpp, z};
    double x[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        x[r] = 0.0;
        x[r] += P.so[3 * r + 0] * xin[0];
        x[r] += P.so[3 * r + 1] * xin[1];
        x[r] += P.so[3 * r + 2] * xin[2];
    }
    const double i0 = x[0] * P.pixels_per_km, j0 = x[1] * P.pixels_per_km;
    if (!(fabs(i0) < n && fabs(j0) < n)) return false;
    const int im = iround_(i0), jm = iround_(j0);
    const long long q = (long long)(im + n) * side + (jm + n);
    if (fac == FI[q] || !(ZI[q] > -0.99 * SHAPE_HUGENUMBER)) return false;
    return posmask_zill(ZI, n, side, i0, j0, im, jm) - x[2] > P.mask_tol;
}

// MODE RASTER_RADAR: radar views, shading and delay-Doppler synthesis; POS maps
// only when a.keep_pos asks for them. RASTER_SUN (double only, as the next two):
// sun views, depth and facet maps; nothing reads their cosines, so nothing is
// shaded. RASTER_PHOTO: the observer views of lightcurve points and sky frames,
// after their sun views: shading, shadows, photometry and POS maps; a tile's
// brightness goes to a.lc_part (as a kernel of its own, which read the maps
// back, photometry took 0.70 ms on 800 points). RASTER_POS: single POS views,
// shading and POS maps on top of what the images hold. 800 points' sun and
// observer launches took 1.63 ms while sun views and single views were one
// kernel, 1.52 apart (no spills, no shading) and 1.38 with the resident warps
// that this allows.
template <typename T, int MODE> __host__ __device__ constexpr int raster_warps()
{
    return MODE == RASTER_SUN || MODE == RASTER_PHOTO ? RASTER_WARPS_MAPS
         : sizeof(T) == 4 ? RASTER_WARPS_F32 : RASTER_WARPS_F64;
}
// FEW_VIEWS: bins of at most FEW entries are not listed.
template <typename T, int NT, int MODE, bool FEW_VIEWS>
__global__ void __launch_bounds__(NT, raster_warps<T, MODE>() * 32 / NT)
k_raster(const __grid_constant__ RasterArgs a)
{
    grid_dep_trigger();
    grid_dep_wait();
    constexpr int PP = TILE_PIX / NT;          // pixels per thread
    constexpr bool MAPS = MODE != RASTER_RADAR, SUN = MODE == RASTER_SUN, PHOTO = MODE == RASTER_PHOTO;
    constexpr bool accumulate = MODE == RASTER_POS;
    __shared__ TileShared<T, NT> sh;
    // radar views: the shaded pixels' depth and cos(e)
    __shared__ double pz[MAPS ? NT / 32 : TILE_PIX];
    __shared__ T pc[MAPS ? 1 : TILE_PIX];
    const int tid = threadIdx.x, lane = tid & 31;

    for (int w = blockIdx.x; w < a.nwork; w += gridDim.x) {
        const int4 item = a.work[w];
        const int tile = item.y, ti0 = item.z, tj0 = item.w;
        const int2 *bin = a.bin_ids + (size_t)tile * a.cap;
        const int count = a.bin_count[tile];
        const FrameGeom &g = a.geoms[item.x];
        const bool writes_pos = MAPS || a.keep_pos;
        if (count == 0 && !writes_pos) continue;
        const int n = g.n;
        const bool smooth = g.smooth != 0;
        const double4 *vt = static_cast<const double4 *>(a.vt) + g.vt_base;

        if (MAPS && count == 0) {
            // nothing here: the background, without the phases and barriers
            for (int r = 0; r < PP; r++) {
                const int p = tid + r * NT, pi = ti0 + p / TILE_W, pj = tj0 + p % TILE_W;
                if (pi > n || pj > n) continue;
                const long long q = g.pos_base + (long long)(pi + n) * g.side + (pj + n);
                if constexpr (accumulate) {
                    a.won[q] = 0;
                    continue;
                }
                static_cast<double *>(a.pos_z)[q] = -SHAPE_HUGENUMBER;
                a.pos_f[q] = -1;
                if (SUN) continue;
                static_cast<T *>(a.pos_cose)[q] = 0;
                static_cast<T *>(a.pos_cosi)[q] = 0;
                if constexpr (PHOTO) {
                    const long long bb = a.pts[g.frame_index].b_base;
                    if (bb >= 0) a.bimg[bb + (q - g.pos_base)] = 0.0;
                }
            }
            if (PHOTO && tid == 0) a.lc_part[tile] = 0.0;
            continue;
        }
        FrameState &S = a.states[item.x];
        for (int r = 0; r < PP; r++) sh.cnt[tid + r * NT] = 0;
        const double x0 = __dmul_rn((double)ti0, g.kmpp), y0 = __dmul_rn((double)tj0, g.kmpp);
        if (tid < TILE_W) sh.xs[tid] = __dmul_rn((double)(ti0 + tid), g.kmpp);
        else if (tid < 2 * TILE_W) sh.ys[tid - TILE_W] = __dmul_rn((double)(tj0 + tid - TILE_W), g.kmpp);
        else if (tid == 2 * TILE_W) sh.n = 0;
        else if (tid < 2 * TILE_W + 5) sh.cov[tid - 2 * TILE_W - 1] = ((volatile int *)S.cov_i)[tid - 2 * TILE_W - 1];
        else if (!MAPS && tid < 2 * TILE_W + 9)
            sh.lim[tid - 2 * TILE_W - 5] = ((volatile unsigned long long *)S.dellim)[tid - 2 * TILE_W - 5];
        __syncthreads();

        // ---- A: facets to pixels
        bool slow = count > a.cap || count > 65536;      // a candidate is held in 16 bits
        const bool staged = count <= NT, few = FEW_VIEWS && count <= FEW;
        if (!slow) {
            const float ikm = (float)g.ikm;
            for (int k = tid; k < count; k += NT) {
                const int2 e = bin[k];
                const FacetTerms q = facet_terms(vt, a.fvi[e.x]);
                if (staged) store_terms<T, NT>(sh, k, q);
                if (few) few_facet<T, NT>(k, q, e.y, x0, y0, ikm, g.kmpp, sh);
                else bound_facet<T, NT>(k, q, e.y, x0, y0, ikm, g.kmpp, CAND_MORE, sh);
            }
            __syncthreads();
            slow = sh.n > CAND_MORE;
        }
        if (slow)
            tile_chunks<T, NT>(a, g, bin, count, ti0, min(ti0 + TILE_W - 1, n), tj0, min(tj0 + TILE_W - 1, n),
                               smooth && !SUN, sh);      // a sun view has no use for the normal's facet

        double bsum = 0.0;                     // PHOTO: this thread's brightness
        // ---- B: one pixel at a time per thread
        for (int r = 0; r < PP; r++) {
            const int p = tid + r * NT;
            const int li = p / TILE_W, lj = p % TILE_W;
            const int pi = ti0 + li, pj = tj0 + lj;
            const bool inframe = (pi <= n) && (pj <= n);
            const long long q = g.pos_base + (long long)(pi + n) * g.side + (pj + n);
            // an accumulating call's pixel starts from what the images hold
            const bool had = accumulate && inframe && a.pos_f[q] >= 0;
            const double had_z = had ? static_cast<const double *>(a.pos_z)[q] : 0.0;
            // the winner: the largest depth of the facets that cover the
            // pixel, the lowest facet among equals
            PixelHit h = {-1, -1, had_z, 0.0, 0.0, 0.0, 0.0};
            if (slow) {
                h = sh.hit[p];
            } else {
                const double xp = sh.xs[li], yp = sh.ys[lj];
                if (few) sh.cnt[p] = few_candidates<T, NT>(sh, count, li, lj);
                const int nc = candidates<T, NT>(sh, few, p);
                unsigned left = sh.cnt[p];
                for (int i = 0; i < nc; i++) {
                    const int k = candidate<T, NT>(sh, few, p, i, left);
                    FacetTerms q;
                    double s, t;
                    if (k < 0 || !entry_covers<T, NT>(a, vt, bin, sh, staged, k, xp, yp, q, s, t)) continue;
                    const double z = facet_z(q, s, t);
                    const bool first = h.f < 0 && !had;
                    if (!(first || z > h.z || (z == h.z && h.f >= 0))) continue;
                    const int f = bin[k].x;
                    if (first || z > h.z || f < h.f) { h.f = f; h.z = z; h.s = s; h.t = t; }
                }
                h.gf = h.f; h.gs = h.s; h.gt = h.t;
            }
            const bool covered = h.f >= 0;
            {
                // covered-pixel bbox (POSrect with (i,i,j,j),
                // posvis.c:278-280): a warp's ballot holds two rows of the
                // tile; an atomic only where it can move the frame's value
                const unsigned b = __ballot_sync(0xffffffffu, covered);
                if (lane == 0 && b) {
                    const unsigned cols = (b | (b >> 16)) & 0xffffu;
                    const int i0 = pi + ((b & 0xffffu) ? 0 : 1), i1 = pi + ((b >> 16) ? 1 : 0);
                    const int j0 = tj0 + __ffs(cols) - 1, j1 = tj0 + 31 - __clz(cols);
                    if (i0 < sh.cov[0]) atomicMin(&S.cov_i[0], i0);
                    if (i1 > sh.cov[1]) atomicMax(&S.cov_i[1], i1);
                    if (j0 < sh.cov[2]) atomicMin(&S.cov_j[0], j0);
                    if (j1 > sh.cov[3]) atomicMax(&S.cov_j[1], j1);
                }
            }
            const bool bistatic_obs = PHOTO || (accumulate && g.kind == VIEW_LC_OBS);
            // nothing reads the sun view's cosines of a lightcurve or sky frame
            const bool shade = !SUN && covered;
            const double z = covered ? h.z : -SHAPE_HUGENUMBER;
            const int fac = h.f;
            T cosa = 0, cosb = 0;
            if (accumulate && inframe) {
                cosa = static_cast<const T *>(a.pos_cose)[q];
                if (g.kind != VIEW_LC_SUN) cosb = static_cast<const T *>(a.pos_cosi)[q];
            }
            if (shade) {
                T r0 = 0, r1 = 0, r2 = 0;
                auto normal = [&]() {
                    if (sizeof(T) == 8 || !smooth) {
                        double m[3];
                        body_normal64(a, h.gf, h.gs, h.gt, smooth, m);
                        r0 = (T)view_row64(g, 0, m); r1 = (T)view_row64(g, 1, m); r2 = (T)view_row64(g, 2, m);
                    } else {
                        const int4 c = a.fvi[h.gf];
                        const float4 q0 = a.vnf[c.x], q1 = a.vnf[c.y], q2 = a.vnf[c.z];
                        const float s = (float)h.gs, t = (float)h.gt;
                        const float m0 = q0.x + s * (q1.x - q0.x) + t * (q2.x - q1.x);
                        const float m1 = q0.y + s * (q1.y - q0.y) + t * (q2.y - q1.y);
                        const float m2 = q0.z + s * (q1.z - q0.z) + t * (q2.z - q1.z);
                        r0 = g.foa[0] * m0 + g.foa[1] * m1 + g.foa[2] * m2;
                        r1 = g.foa[3] * m0 + g.foa[4] * m1 + g.foa[5] * m2;
                        r2 = g.foa[6] * m0 + g.foa[7] * m1 + g.foa[8] * m2;
                    }
                };
                if (h.gf >= 0) normal();
                if (smooth && !slow) {
                    // FP32 form: a view-z component within its rounding of
                    // zero (normals of unit size, s and t below 1) takes its
                    // sign in FP64
                    bool faces = r2 > (T)0;
                    if (sizeof(T) == 4 && fabs(r2) <= (T)4e-6) {
                        double m[3];
                        body_normal64(a, h.f, h.s, h.t, true, m);
                        faces = view_row64(g, 2, m) > 0.0;
                    }
                    if (!faces) {
                        const PixelHit c = pixel_history<T, NT, FEW_VIEWS>(a, g, bin, count, sh, p, h.f, had, had_z);
                        h.gf = c.gf; h.gs = c.gs; h.gt = c.gt;
                        if (h.gf >= 0) normal();
                    }
                }
                if (h.gf >= 0) {
                    if (smooth) {
                        const T norm = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
                        if (norm != (T)0) {
                            r2 /= norm;
                            if (bistatic_obs) { r0 /= norm; r1 /= norm; }
                        }
                    }
                    if (r2 > (T)0) {
                        cosa = r2;
                        if (bistatic_obs) {
                            cosb = r0 * (T)g.usrc[0] + r1 * (T)g.usrc[1] + r2 * (T)g.usrc[2];
                            if (cosb <= (T)0) cosa = 0;
                        }
                    }
                }
            }
            if constexpr (PHOTO) {
                const LcPointDev &P = a.pts[g.frame_index];
                if (cosa != 0.0) {
                    if (photo_shadowed(a, g, P, pi, pj, z, fac)) cosa = 0.0;
                    if (a.mark_seen && cosa > a.mincosine_seen && cosb > a.mincosine_seen) a.seen[fac] = 1;
                }
                const double b = (covered && cosa > 0.0 && cosb > 0.0) ? photo_brightness(P, cosa, cosb) : 0.0;
                bsum += b;
                // a sky frame keeps its brightness image (pos->b of apply_photo)
                if (P.b_base >= 0 && inframe) a.bimg[P.b_base + (q - g.pos_base)] = b;
            }
            if (writes_pos && inframe) {
                double *Z = static_cast<double *>(a.pos_z);
                T *CE = static_cast<T *>(a.pos_cose), *CI = static_cast<T *>(a.pos_cosi);
                if (accumulate) {
                    a.won[q] = covered ? 1 : 0;
                    if (covered) { Z[q] = z; a.pos_f[q] = fac; }
                } else {
                    Z[q] = z;
                    a.pos_f[q] = fac;
                }
                if (!SUN) CE[q] = cosa;   // cos(i) in a sun view (pos->cosill)
                if (!SUN && g.kind != VIEW_LC_SUN) CI[q] = cosb;
            }
            if constexpr (!MAPS) {
                if (covered && a.mark_seen && !g.no_seen && (double)cosa > a.mincosine_seen) a.seen[fac] = 1;
                pz[p] = z;
                pc[p] = covered ? cosa : (T)0;
            }
        }

        if constexpr (PHOTO) {
            // the tile's brightness, in a fixed order
            for (int off = 16; off > 0; off >>= 1) bsum += __shfl_down_sync(0xffffffffu, bsum, off);
            if (lane == 0) pz[tid >> 5] = bsum;
            __syncthreads();
            if (tid == 0) {
                double v = 0.0;
                for (int k = 0; k < NT / 32; k++) v += pz[k];
                a.lc_part[tile] = v;
            }
        }

        // ---- C: delay-Doppler synthesis on a scattered pixel-to-thread map.
        // Neighbouring pixels share facets, which phase B's loads want, but
        // they hit the same delay-Doppler bins, so a compact warp's atomics
        // would repeat addresses within one instruction.
        if constexpr (!MAPS) {
            __syncthreads();
            for (int r = 0; r < PP; r++) {
                const int p = ((tid + r * NT) * 37 + 11) & (TILE_PIX - 1);
                const int pi = ti0 + p / TILE_W, pj = tj0 + p % TILE_W;
                const T cosa = pc[p];
                const bool lit = cosa > (T)0;
                PixPos pp = {0.0, 0.0};
                PixDD<T> dd;
                dd.ok = false;
                if (lit) {
                    if constexpr (sizeof(T) == 4) dd = pixel_dd_setup_x(g, pi, pj, pz[p], pp);
                    else dd = pixel_dd_setup(g, pi, pj, pz[p], pp);
                }
                // delay / Doppler extremes of the frame's lit pixels as dkey
                // keys: reduced and added only by a warp that holds a value
                // outside the frame's current extremes
                const unsigned long long kd = dkey(pp.del), kp = dkey(pp.dop);
                const bool out = lit && (kd < sh.lim[0] || kd > sh.lim[1] || kp < sh.lim[2] || kp > sh.lim[3]);
                if (__any_sync(0xffffffffu, out)) {
                    const unsigned long long k0 = warp_kmin(lit ? kd : ~0ull), k1 = warp_kmax(lit ? kd : 0ull);
                    const unsigned long long k2 = warp_kmin(lit ? kp : ~0ull), k3 = warp_kmax(lit ? kp : 0ull);
                    if (lane == 0) {
                        int l[4];
                        dd_bin_limits(g, dkey_inv(k0), dkey_inv(k1), dkey_inv(k2), dkey_inv(k3), l);
                        atomicMin(&S.idellim[0], l[0]); atomicMax(&S.idellim[1], l[1]);
                        atomicMin(&S.idoplim[0], l[2]); atomicMax(&S.idoplim[1], l[3]);
                        atomicMin(&S.dellim[0], k0); atomicMax(&S.dellim[1], k1);
                        atomicMin(&S.doplim[0], k2); atomicMax(&S.doplim[1], k3);
                    }
                }
                // The footprint goes straight to the frame's fit image in HBM:
                // FP32 as 16-byte vector reductions, FP64 as scalar atomics
                // (both measured faster than a shared-memory accumulator
                // flushed per tile).
                T *fit = static_cast<T *>(a.fit) + g.fit_base;
                T *row = sh.stage[tid].w;
                if (g.dop1d) {
                    // a spectrum is summed in FP64 in both forms
                    double *spec = (sizeof(T) == 4 ? a.fit64 : static_cast<double *>(a.fit)) + g.fit_base;
                    const bool staged_px = dd.ok && stage_fits(g, dd);
                    const T amp = staged_px ? stage_pixel<T>(a, g, cosa, dd, row) : (T)0;
                    __syncwarp();
                    const unsigned mask = __ballot_sync(0xffffffffu, staged_px);
                    const int c1 = warp_min(staged_px ? dd.idop_min : INT_MAX);
                    const int c2 = warp_max(staged_px ? dd.idop_max : INT_MIN);
                    add_spectra<T, double>(mask, dd.idop_min, amp, c1, c2, &sh.stage[tid & ~31], spec);
                    __syncwarp();
                    if (dd.ok && !staged_px) {
                        pixel_dd_scatter<T, double>(a, g, cosa, dd, spec);
                    } else if (lit && !dd.ok) {
                        S.any_overflow = 1;
                        pixel_dop_overflow<T>(a, g, cosa, dd);
                    }
                } else if (dd.ok && !pixel_dd_scatter_lean<T>(a, g, cosa, dd, fit)) {
                    if (stage_fits(g, dd)) {
                        const T amp = stage_pixel<T>(a, g, cosa, dd, row);
                        scatter_staged<T>(g, dd, amp, row, fit);
                    } else {
                        pixel_dd_scatter<T, T>(a, g, cosa, dd, fit);
                    }
                }
            }
        }
        __syncthreads();
    }
}

// variant 0: 256 threads per tile; 1: 128 (two pixels a thread, smaller CTAs).
// f(kernel, threads) for the kernel that a's mode and variant select (a single
// POS view is one launch of a few tiles: 256 threads).
template <typename T, int MODE, typename F>
inline void with_raster_kernel_of(const RasterArgs &a, F f)
{
    if (a.variant == 1 && MODE != RASTER_POS)
        return a.few ? f(k_raster<T, 128, MODE, true>, 128) : f(k_raster<T, 128, MODE, false>, 128);
    return a.few ? f(k_raster<T, 256, MODE, true>, 256) : f(k_raster<T, 256, MODE, false>, 256);
}
template <typename T, typename F>
inline void with_raster_kernel(const RasterArgs &a, F f)
{
    if constexpr (sizeof(T) == 8) {
        if (a.mode == RASTER_SUN) return with_raster_kernel_of<T, RASTER_SUN>(a, f);
        if (a.mode == RASTER_POS) return with_raster_kernel_of<T, RASTER_POS>(a, f);
        if (a.mode == RASTER_PHOTO) return with_raster_kernel_of<T, RASTER_PHOTO>(a, f);
    }
    return with_raster_kernel_of<T, RASTER_RADAR>(a, f);
}

template <typename T>
inline void launch_raster_t(const RasterArgs &a, cudaStream_t s)
{
    if (a.nwork <= 0) return;
    const int grid = (a.grid > 0 && a.grid < a.nwork) ? a.grid : a.nwork;
    with_raster_kernel<T>(a, [&](auto kern, int nt) { launch_k(kern, dim3(grid), dim3(nt), 0, s, a.pdl != 0, a); });
}

// Called once per device before any launch (not inside stream capture).
template <typename T>
inline cudaError_t configure_raster_t()
{
    cudaError_t e = cudaSuccess;
    RasterArgs a = {};
    for (a.mode = RASTER_RADAR; a.mode <= (sizeof(T) == 8 ? RASTER_POS : RASTER_RADAR); a.mode++)
        for (int k = 0; k < 4 && e == cudaSuccess; k++) {
            a.variant = k & 1;
            a.few = k >> 1;
            with_raster_kernel<T>(a, [&](auto kern, int) {
                e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, RASTER_SHARED_PCT);
            });
        }
    return e;
}

// Resident CTAs per SM of the kernel launch_raster_t would launch for a
// (0 when the query fails): the persistent grid is this times the SM count.
template <typename T>
inline int raster_occupancy_t(const RasterArgs &a)
{
    int n = 0;
    cudaError_t e = cudaSuccess;
    with_raster_kernel<T>(a, [&](auto kern, int nt) { e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, nt, 0); });
    return e == cudaSuccess ? n : 0;
}

}  // namespace shape
