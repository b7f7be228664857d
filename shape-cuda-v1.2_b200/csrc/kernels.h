// Kernel launchers of the SHAPE B200 engine (implemented in core.cu,
// raster_f64.cu, raster_f32.cu). All launches take the engine stream.
#pragma once

#include <cuda_runtime.h>

#include "engine_internal.h"
#include "shape_b200.h"

namespace shape {

// Programmatic dependent launch (batched forms): a kernel launched with
// launch_k(..., pdl = true) may be scheduled before the previous kernel on
// its stream has finished, and waits in grid_dep_wait, before its first access
// to that kernel's outputs, until it has (a no-op after an ordinary launch).
// grid_dep_trigger at a kernel's start lets the next one's blocks become
// resident once every block of this one has started, so they take no slots
// from it and the launch latency between the two is hidden. Kernel k + 2 needs
// no trigger of kernel k's: kernel k + 1 finishes only after its own wait.
#ifdef __CUDACC__
__device__ __forceinline__ void grid_dep_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

template <typename... KArgs, typename... Args>
inline void launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl,
                     Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? at : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

// Per-component transform of a model with several components: the rotation
// matrix (9, row-major), the translation (3), whether to rotate and whether
// to translate (nonzero offsets), two spare slots.
constexpr int CXF_N = 16;

struct ModelDev {
    int nv, nf;
    const double *a, *u, *r, *scale;   // a,u: [nv*3]; scale: 3 per component
    const int *vcomp;                  // [nv] component of each vertex (null: one component)
    const double *cxf;                 // [ncomp * CXF_N] component transforms (null: one component)
    const int *fv;                     // [nf*3]
    const int *af_ptr, *af_idx;
    double4 *vx, *vn, *fn;             // realized
    float4 *vnf;                       // vertex normals rounded to float (FP32 form; may be null)
    double *area;
    int4 *fvi;                         // corner indices, padded
};

// What a raster launch does with its views (k_raster).
enum { RASTER_RADAR, RASTER_SUN, RASTER_PHOTO, RASTER_POS };

struct RasterArgs {
    const FrameGeom *geoms;
    // tiles: (view, index of the tile among all views', first pixel row, first
    // pixel column); with the last three here, the tile's bin is read without
    // waiting for the view's constants
    const int4 *work;
    int nwork;                 // items
    int grid;                  // CTAs (0: one per item); fewer CTAs stride over the rest
    int pdl;                   // programmatic dependent launch (launch_k)
    const void *vt;            // double4 view-frame vertices (both forms)
    const int4 *fvi;
    const double4 *vn;
    const float4 *vnf;
    const double4 *fn;
    int nf;
    const int *bin_count;
    const int2 *bin_ids;        // (facet, tile-relative bbox) entries
    int cap;
    FrameState *states;
    const RadarLawDev *laws;
    void *fit;                 // T image arena (radar views)
    double *fit64;             // FP32 form: FP64 sums of the one-row (Doppler) frames, at their fit offsets
    void *pos_z, *pos_cose, *pos_cosi;  // POS maps: z double, cos(e) / cos(i) T (keep_pos or lightcurves)
    int *pos_f;
    unsigned char *seen;
    double mincosine_seen;
    int mark_seen;
    int keep_pos;
    double *ovf;               // Doppler overflow spectra (DOP_MAXOVERFLOW per Doppler frame)
    // FP64 raster of a single view into images that already hold earlier
    // calls' results (posvis accumulating over model components): each pixel
    // starts from its z / facet / cos(e) / cos(i), and won[p] is set to 1
    // where this launch assigned pixel p. 0 for the engine's evaluations.
    int accumulate;
    unsigned char *won;
    int variant;               // 0: 256 threads per tile, 1: 128
    int few;                   // 1: the kernel for views of few facets per tile (raster_few)
    int mode;                  // RASTER_*
    // RASTER_PHOTO: the views' points, the tiles' brightness sums and the
    // brightness images of sky frames (LcPointDev::b_base)
    const LcPointDev *pts;
    double *lc_part;
    double *bimg;
};

// core.cu (FP64, no FMA contraction)
void launch_realize(const ModelDev &m, cudaStream_t s);      // launch_realize_vf + launch_realize_vn
void launch_realize_vf(const ModelDev &m, cudaStream_t s);   // vertices, facet normals and areas
void launch_realize_vn(const ModelDev &m, cudaStream_t s);   // vertex normals (after _vf)

// Model sums for the penalty terms (penalty.cu), in this order.
// The sums run over the model's active facets, edges and vertices: all of
// them for one component; for several, those check_surface leaves active
// (not inside another component), with the counts of active edges and
// vertices and check_surface's error flag (an edge-crossing list overflow).
enum {
    MSUM_VOLUME, MSUM_COM, MSUM_IXX = MSUM_COM + 3, MSUM_IYY, MSUM_IZZ, MSUM_IXY, MSUM_IXZ, MSUM_IYZ,
    MSUM_NONSMOOTH, MSUM_CONCAVITY, MSUM_RDEV, MSUM_RDEV_MAX, MSUM_NSIDES, MSUM_NVERT, MSUM_SURF_ERR, MSUM_N
};
struct ModelSumArgs {
    ModelDev m;                 // realized model (vx, fn, fv, u, r, scale, vcomp)
    const int4 *sides;          // edges: (end vertex v1, f1's third vertex, f1, f2)
    const int *side_v2;         // the edges' other end vertices (several components)
    int nsides;
    int ncomp;
    const int2 *comp_facets;    // [ncomp] (first facet, facets) of each component
    unsigned char *act_v, *act_f;   // check_surface's flags (null: one component, all active)
    int *surf_err;              // check_surface's error flag (zeroed before it runs)
    double *part;               // [model_sums_blocks() * MSUM_N]
    double *out;                // [MSUM_N]
};
int model_sums_blocks();
void launch_model_sums(const ModelSumArgs &a, cudaStream_t s);   // two launches
void launch_check_surface(const ModelSumArgs &a, cudaStream_t s);   // several components: the active flags
void launch_reset_state(FrameState *st, int nviews, int *bin_count, int ntiles, cudaStream_t s);
// pdl: programmatic dependent launch (launch_k)
void launch_xform_f64(const FrameGeom *g, int nviews, const double4 *vx, int nv, double4 *vt,
                      cudaStream_t s, bool pdl = false);
// the first launch of a batched evaluation (k_front)
struct FrontArgs {
    static constexpr int CLEARS = 7;
    const FrameGeom *geoms;
    int nviews;
    ModelDev m;
    double4 *vt;
    FrameState *blank;                 // states to blank
    // binning within the launch (bin_ids null: a launch of its own follows):
    // into states and counts that an earlier launch has blanked
    FrameState *states;
    int *bin_count;
    int2 *bin_ids;
    int cap;
    // parameter changes since the device arrays were last written: the scale
    // factors (of up to SCALES / 3 components) and up to CHANGES deviations
    // travel with the launch, which also stores them, instead of a copy of all
    // of them ahead of it (5 us before the first kernel could start)
    static constexpr int SCALES = 24, CHANGES = 8;
    double scale[SCALES];
    int nscale;                        // 0: the arrays hold the parameters
    int nchange, change_at[CHANGES];
    double change_to[CHANGES];
    double *r_out, *scale_out;
    unsigned char *clear[CLEARS];      // arrays to clear (16-byte aligned) and their bytes
    size_t clear_bytes[CLEARS];
    int views;                         // views whose vertices a thread writes
    int nb_bin, nb_vn, nb_xform, nb_model;   // blocks of the first ranges (set by launch_front)
};
void launch_front(const FrontArgs &a, cudaStream_t s);
// the vertex normals as extra blocks of k_bin (nv 0: none)
struct VnormalArgs {
    int nv;
    const int *af_ptr, *af_idx;
    double4 *vn;
    float4 *vnf;
};
void launch_bin_f64(const FrameGeom *g, int view0, int nviews, const ModelDev &m, const double4 *vt,
                    FrameState *st, int *bin_count, int2 *bin_ids, int cap, cudaStream_t s, bool pdl = false,
                    bool vnormals = false);

// Chi-square items: (frame, share of its lit box) or (frame, -1) for its
// geometry results, one block each.
struct Chi2Args {
    const int2 *items;
    int nitems;
    const double *obs, *oov;
    void *fit;                   // double or float
    const double *fit64;         // FP32 form: the Doppler frames' FP64 sums
    double *partials;            // [nitems * 4]: m2, om + compensations
    const double *o2;            // [nframes * 2]: sum obs^2 / var and its compensation (launch_frame_o2)
};
struct FrameHost {             // per radar frame constants for finalize
    double weight, dof, cal_in;
    int cal_floating, badradar;
    double badradar_logfactor;
    int view;
    int set;
    int item0, nitems;
    int dop_index;             // Doppler frame: index of its overflow terms, else -1
    double sdev;               // Doppler frame: receiver noise sdev (overflow variance)
    // smeared frames (src/shape/calc_fits.c:475-594): views, whether any
    // view's footprint was too wide, and the sum of those views'
    // badradar log-factors (the objective adds dof * sum / views); the
    // frame's own badradar and badradar_logfactor are its epoch view's
    int nviews;
    int badradar_any;
    double badradar_lfsum;
};
struct FinalizeArgs {
    int nframes;
    const FrameHost *fh;
    const FrameGeom *geoms;
    const FrameState *states;
    shape_deldop_result *results;
    const double *set_delpp, *set_doppp;     // per set del/dop per pixel
    const double *dop_extra;                 // per frame
    const double *ovf;                       // overflow spectra
    double *ovf_out;                         // per Doppler frame: DOP_OVF_TERMS values
};

// Doppler overflow terms per Doppler frame (src/shape/pos2doppler.c:451-499):
// o2, m2, xsec, mean bin, and the badradar flag and log-factor of a model wider
// than the overflow spectrum.
constexpr int DOP_OVF_TERMS = 6;
// sum obs^2 / var of each radar frame (partials: as Chi2Args's, scratch here)
void launch_frame_o2(const int2 *items, int nitems, const FrameHost *fh, int nframes, const FrameGeom *geoms,
                     const double *obs, const double *oov, double *partials, double *o2, cudaStream_t s);

struct LcSetDev {
    int npts, n;                // calc points, observed points
    int pt0;                    // first calc point (global)
    const double *x, *t, *obs, *oov;  // device arrays
    // the spline's elimination, which depends on the epochs only: the lower
    // coefficients w, the pivots and their reciprocals, the multipliers of
    // y2[i+1] in y2[i] and the spans ([5 * npts])
    const double *spl;
    double *y, *y2, *fit;       // device outputs
    double *scratch;            // work arrays of a set too large for shared memory (null: none)
    double o2;                  // sum obs^2 / var in order
    double weight, dof, cal_in;
    int cal_floating;
};
struct LcFinalizeArgs {
    int nsets;
    const LcSetDev *sets;
    const LcPointDev *pts;
    const FrameGeom *geoms;
    const FrameState *states;
    const double *tile_part;    // brightness of each tile (RASTER_PHOTO)
    double *set_out;            // per set: cal, chi2, posbnd flag, logfactor sum
    size_t smem_per_set;        // dynamic shared memory (lc_finalize_smem of the largest set), 0: global
};
constexpr size_t LC_FINALIZE_SMEM_MAX = 160 * 1024;
size_t lc_finalize_words(int npts, int n);   // doubles of a set's work arrays
size_t lc_finalize_smem(int npts, int n);
cudaError_t configure_lc_finalize();
void launch_lc_finalize(const LcFinalizeArgs &a, cudaStream_t s, bool pdl);

// Spin realization inside an evaluation (spin.cu; principal-axis
// rotators): one thread per radar frame (its epoch view) or lightcurve point
// realizes ae (and a frame's spin vector) from the device spin state and
// its dataset's offsets, then the view constants as the host sets them.
struct SpinViewSrc {
    int kind;                   // 0 radar frame, 1 lightcurve point
    int index;                  // global radar frame or point index
    int rec;                    // dataset record: offsets at off[6 rec ..]
    int dd;                     // delay-Doppler set of a radar frame
    double t;                   // epoch (light-time corrected)
    double orb[3];              // orbital spin contribution (radar frames)
};
struct SpinRealizeArgs {
    int n;
    const SpinViewSrc *src;
    const shape_spin_state *spin;
    const double *off;                 // per record: angleoff[3], omegaoff[3]
    shape_deldop_frame *frames;        // ae and spin written
    const shape_deldop_set *ddsets;
    shape_lghtcrv_point *points;       // ae written
    FrameGeom *geoms;
    FrameHost *fh;
    double *dop_extra;
    LcPointDev *lcpts;
};
void launch_realize_views(const SpinRealizeArgs &a, cudaStream_t s);

struct SetRec { int type; int first; int count; };   // type 0 deldop (frames), 1 lightcurve (set index), 2 plane-of-sky (frames)

// Plane-of-sky frames (calc_poset after apply_photo, and chi2_poset): blocks
// blocks per frame resample the brightness image onto the fit grid,
// checks that the grid holds every lit pixel and forms the chi-square.
constexpr int POSET_PART = 8;
struct PosetArgs {
    int nframes;
    const PosetFrameDev *frames;
    const LcPointDev *pts;
    const FrameGeom *geoms;
    const FrameState *states;
    const double *bimg;         // brightness images
    const double *obs, *oov;    // observed images and 1/variance
    double *fit;                // fit images
    shape_poset_result *res;    // per-frame results
    int blocks;                 // blocks per frame
    double *part;               // [nframes * blocks * POSET_PART] their sums and extremes
    int *counters;              // [nframes] finished blocks, zero before the launch
};
void launch_poset_frames(const PosetArgs &a, cudaStream_t s, bool pdl);
struct SummaryArgs {
    int nsets;
    const SetRec *sets;
    const FrameHost *fh;
    const shape_deldop_result *results;
    const double *lc_out;       // per lightcurve set: cal, chi2, posbnd, logfactor sum
    const double *lc_dof;
    const double *lc_npts;
    const shape_poset_result *ps_res;   // plane-of-sky frames' results
    const PosetFrameDev *ps_frames;
    double dof_poset;           // plane-of-sky dof (calc_fits.c:408)
    double dof, dof_radar;      // all data / delay-Doppler + Doppler (calc_fits.c:409)
    double bad_objfactor;
    int baddiam;
    double baddiam_logfactor;
    shape_eval_summary *out;
};
// Radar frames' chi-square, results and the totals; counters: nframes + 1 ints,
// zero before the launch
void launch_chi2_summary(const Chi2Args &ca, const FinalizeArgs &fa, const SummaryArgs &sa, int *counters,
                         int fp32, cudaStream_t s, bool pdl);
// the totals alone (no radar frames)
void launch_totals(const SummaryArgs &a, cudaStream_t s, bool pdl);

// Whether tiles of this many bin entries in all are rastered by the kernels for
// few facets per tile (raster_impl.cuh, FEW): where the tiles that have any hold
// RASTER_FEW_MEAN on average.
constexpr int RASTER_FEW_MEAN = 24;
inline int raster_few(long long entries, long long tiles) { return tiles > 0 && entries <= RASTER_FEW_MEAN * tiles; }
// raster_f64.cu / raster_f32.cu
void launch_raster_f64(const RasterArgs &a, cudaStream_t s);
void launch_raster_f32(const RasterArgs &a, cudaStream_t s);
// resident CTAs per SM of the raster kernel these arguments select
int raster_occupancy_f64(const RasterArgs &a);
int raster_occupancy_f32(const RasterArgs &a);
cudaError_t configure_raster_f64();
cudaError_t configure_raster_f32();

}  // namespace shape
