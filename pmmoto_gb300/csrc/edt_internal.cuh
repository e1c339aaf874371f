// Internal interface between the EDT kernels and their users (morphology).
#pragma once

#include <cfloat>
#include <climits>
#include <cmath>

#include "pmg_common.cuh"

namespace pmg {

// Imported boundary hulls per side the envelope kernels hold (the reference
// keeps at most num_hull + 1 = 5); entry points accept num_hull + 1 <= kMaxHull.
constexpr int kMaxHull = 8;

// Lines of a pass: all lines along axis `ax` whose coordinates on the other
// two axes (d1 < d2) lie in [b1lo, b1lo + nb1) x [b2lo, b2lo + nb2).
struct Lines {
    long long s0, s1, s2;
    int ax;
    int b1lo, nb1, b2lo, nb2;
    __host__ __device__ long long count() const { return (long long)nb1 * nb2; }
};

struct LineGeo {
    long long base, stride;
    int n;
    int a, b; // coordinates of the line along the two other axes (d1 < d2)
};

__device__ __forceinline__ LineGeo line_addr(const Lines &L, long long li)
{
    LineGeo g;
    const int a = L.b1lo + (int)(li / L.nb2);
    const int b = L.b2lo + (int)(li - (li / L.nb2) * L.nb2);
    g.a = a;
    g.b = b;
    if (L.ax == 0) { // lines over (j, k)
        g.base = (long long)a * L.s2 + b;
        g.stride = L.s1 * L.s2;
        g.n = (int)L.s0;
    } else if (L.ax == 1) { // lines over (i, k)
        g.base = (long long)a * L.s1 * L.s2 + b;
        g.stride = L.s2;
        g.n = (int)L.s1;
    } else { // lines over (i, j)
        g.base = ((long long)a * L.s1 + b) * L.s2;
        g.stride = 1;
        g.n = (int)L.s2;
    }
    return g;
}

// Heights as they are, or as counts of voxels (0x4000 and more: none).
__device__ __forceinline__ float height_of(const float *p, float) { return __ldg(p); }
__device__ __forceinline__ float height_of(const uint16_t *p, float res)
{
    const uint32_t c = __ldg(p);
    const float d = fmul((float)c, res);
    return c >= 0x4000u ? FLT_MAX : fmul(d, d);
}


__host__ inline Lines all_lines(const int64_t *shape, int ax)
{
    Lines L;
    L.s0 = shape[0];
    L.s1 = shape[1];
    L.s2 = shape[2];
    L.ax = ax;
    const int d1 = ax == 0 ? 1 : 0, d2 = ax == 2 ? 1 : 2;
    L.b1lo = 0;
    L.nb1 = (int)shape[d1];
    L.b2lo = 0;
    L.nb2 = (int)shape[d2];
    return L;
}

// Fused morphology epilogue of the last envelope pass (addition/subtraction,
// src/pmmoto/filters/morphological_operators.py:103-228): the distance is
// square-rooted as np.sqrt does, compared with the radius in the precision
// numpy would use, the extension halo is cut off (utils.unpad) and wall
// planes are forced to 0 (set_wall_bcs).
struct MorphEpi {
    uint8_t *out;         // unextended volume (o0, o1, o2)
    long long o0, o1, o2; // unextended shape
    int e0, e1, e2;       // low-side extension per axis
    int wall[6];          // wall planes: axis0 lo/hi, axis1 lo/hi, axis2 lo/hi
    float lim;            // largest squared distance within the radius (within_limit)
    int dilate;           // 1: addition (1 where d <= r), 0: subtraction
};

// The largest float v that the reference's comparison counts as within: thr_sq
// >= 0 (FFT-ball modes): v <= thr_sq; else sqrt(v) <= r, the float root compared
// in float64 (cmp64, a numpy float64 radius) or with r rounded to float.  The
// root is monotone, so kernels compare the squared distance alone (the float64
// comparison was 28 of 45 us of an erosion of 200^3 voxels).
float within_limit(double r, int cmp64, double thr_sq);

// Store of the fused morphology epilogue: "distance within the radius" at
// position i of line g (extended coordinates) -> 0/1 of the unextended volume.
__device__ __forceinline__ void morph_put(const MorphEpi &me, const LineGeo &g, int i, bool within)
{
    const long long io = g.a - me.e0, jo = g.b - me.e1;
    const int ko = i - me.e2;
    if (ko < 0 || ko >= me.o2)
        return;
    uint8_t v = me.dilate ? (uint8_t)within : (uint8_t)!within;
    if ((me.wall[0] && io == 0) || (me.wall[1] && io == me.o0 - 1) || (me.wall[2] && jo == 0) ||
        (me.wall[3] && jo == me.o1 - 1) || (me.wall[4] && ko == 0) || (me.wall[5] && ko == me.o2 - 1))
        v = 0;
    me.out[(io * me.o1 + jo) * me.o2 + ko] = v;
}

// The threshold of the epilogue on a squared distance `val`.
__host__ __device__ __forceinline__ bool morph_within(const MorphEpi &me, float val) { return val <= me.lim; }

__device__ __forceinline__ void morph_store(const MorphEpi &me, const LineGeo &g, int i, float val)
{
    morph_put(me, g, i, morph_within(me, val));
}

// Lines the exact streaming kernel hands back to the general one carry a
// marker in their first output: NaN (float forms) or 255 (morphology).
__device__ __forceinline__ bool line_marked(const float *fout, const MorphEpi &me, const LineGeo &g, int form)
{
    if (form == PMG_EDT_MORPH) {
        const long long io = g.a - me.e0, jo = g.b - me.e1;
        return me.out[(io * me.o1 + jo) * me.o2] == 255;
    }
    const float v = fout[g.base];
    return v != v;
}

// cap: heights above cap * res^2 are treated as absent and outputs above it
// are written as FLT_MAX (INT_MAX: no cap).
int launch_envelope_exact(const float *fin, float *fout, const Lines &Ls, float res, int form,
                          const MorphEpi &me, cudaStream_t st, int cap);
bool exact_path_ok(float res, const pmg_axis_cfg &cfg, int n);
// Largest integer T < lim with morph_within(T * a) (the threshold is monotone
// in the squared distance), -1 when not even 0 is within, lim when T >= lim.
int morph_threshold(const MorphEpi &me, float a, int lim);
// Last morphology pass on exact integer heights: within iff E(x) <= T.
int launch_env_thresh(const float *fin, const Lines &Ls, float res, int T, const MorphEpi &me,
                      cudaStream_t st);

// Geometry of an image extended on periodic axes.
struct ExtAxis {
    int periodic;
    int own_lo, own_len; // own region of the padded axis
    int ext_lo;          // low-side extension
    int wall_lo, wall_hi;
    long long S, X;      // padded and extended lengths
};

struct ExtGeo {
    ExtAxis ax[3];
};

__device__ __forceinline__ long long src_index(const ExtAxis &a, long long x, bool &zero)
{
    const long long p = x - a.ext_lo; // coordinate in the padded image
    if (a.periodic) {
        long long q = x - (a.own_lo + a.ext_lo);
        // (mostly within a period on either side: a 64-bit division otherwise)
        if (q < -a.own_len || q >= 2LL * a.own_len)
            q %= a.own_len;
        if (q < 0)
            q += a.own_len;
        else if (q >= a.own_len)
            q -= a.own_len;
        return q + a.own_lo;
    }
    if ((a.wall_lo && p == 0) || (a.wall_hi && p == a.S - 1))
        zero = true;
    return p;
}

// Capped integer morphology (morph_cap.cu): isotropic power-of-two voxels,
// binary image, threshold T <= kCapMaxT; KA, KB: uint16 scratch of the
// extended volume.
constexpr int kCapMaxT = 1023;
bool cap_path_ok(const float *res, const int64_t *X, int T);
// img: the unextended image, read through G (erosions: flag, an int of device
// scratch, tells whether it is binary; when not, *nonbinary is set and nothing
// is written); gate: a device count of the seeds (null: not known to be empty),
// zero making the result all zeros without the envelope passes; xr: a device x
// range of the seed blocks (kRangeBig encoding) -- the result is then written
// only on the x range orange receives ([lo, hi] in whole blocks, lo > hi for
// none) and is undefined elsewhere; rows (dilations without periodic axes): the
// seeds as row words instead of img; rows_out: the result as row words instead
// of bytes (only where cap_rows_out)
int morph_cap_run(const uint8_t *img, const ExtGeo &G, uint16_t *KA, uint16_t *KB, const int64_t *X, int T,
                  const MorphEpi &me, cudaStream_t st, int *flag = nullptr, int *nonbinary = nullptr,
                  const unsigned long long *gate = nullptr, const int *xr = nullptr, int *orange = nullptr,
                  const unsigned *rows = nullptr, unsigned *rows_out = nullptr);
// The last pass can write row words: no extension, line pairs (T small enough).
bool cap_rows_out(const int64_t *X, int T, const MorphEpi &me);
int edt_cap_run(const uint8_t *img, const ExtGeo &G, uint16_t *KA, uint16_t *KB, uint16_t *KC, const int64_t *X, int T,
                int *flag, int *nonbinary, cudaStream_t st);

int launch_pass0(const uint8_t *img, float *out, const Lines &Ls, float res,
                 const pmg_axis_cfg &cfg, cudaStream_t st);
// Longest line of k_lin, and of the envelope passes that hold a line on chip.
constexpr int kLinMaxLine = 2048, kScanMaxLine = 1024;
bool window_path_ok(float res, int n);
// The linear pass along axis 0 (edt_lattice.cu): as counts (>= 0x4000: no
// zero), or as squared distances (no periodic axis).
bool lin_ok(int n, const pmg_axis_cfg &cfg);
int launch_lin_counts(const uint8_t *img, uint16_t *out, const int64_t *shape, const pmg_axis_cfg &cfg,
                      cudaStream_t st);
int launch_lin_float(const uint8_t *img, float *out, const int64_t *shape, float res, const pmg_axis_cfg &cfg,
                     cudaStream_t st);
int launch_linear(const uint8_t *img, float *out, const int64_t *shape, float res, const pmg_axis_cfg &cfg,
                  cudaStream_t st);
// The passes of a transform that run on the integer lattice: cols along axis 1
// (counts: from the counts of the linear pass, whose voxels are 2^shift of its
// own), rows along axis 2; wide1, wide2: finite heights may exceed its range.
struct LatticePlan {
    bool cols, counts, rows, wide1, wide2;
    int shift;
};
LatticePlan lattice_plan(const int64_t *shape, const float *res, const pmg_axis_cfg *cfg);
// (flags: one entry per line)
int lattice_cols(const LatticePlan &P, const void *in, float *out, const int64_t *shape, const float *res,
                 const pmg_axis_cfg *cfg, int num_hull, uint16_t *flags, cudaStream_t st);
int lattice_rows(const LatticePlan &P, const float *in, float *out, const int64_t *shape, const float *res,
                 const pmg_axis_cfg *cfg, int num_hull, int form, uint16_t *flags, cudaStream_t st);
bool cols_capped_ok(const int64_t *X, float res, int T);
int launch_cols_capped(const float *fin, float *fout, const int64_t *X, int lo, int planes, float res, int T,
                       cudaStream_t st);
// Flagged lines: after a lattice pass over heights or counts (of voxels of
// res_height; line_reach), and after a scan (kScanEnds); the whole ones and, when
// the probe chose so, all.
template <class T>
int launch_lattice_ends(const T *fin, float *fout, const Lines &Ls, float res, float res_height, const pmg_axis_cfg &cfg,
                        int num_hull, int form, uint16_t *flag, int defer, cudaStream_t st);
template <class T, class F>
int launch_whole(const T *fin, float *fout, const Lines &Ls, float res, float res_height, const pmg_axis_cfg &cfg,
                 int num_hull, int form, const MorphEpi &me, const F *flag, const int *wide, cudaStream_t st);
constexpr int kWholeLine = 255; // (low byte of a lattice flag)
int launch_ends_float(const float *fin, float *fout, const Lines &Ls, float res, const pmg_axis_cfg &cfg,
                      int num_hull, int form, const MorphEpi &me, const uint8_t *flag, const int *wide,
                      cudaStream_t st);
// Passes whose kernel a probe in front of them chooses (device int, null: no
// probe; nonzero: the float envelope takes every line) start while the probe
// still runs: their first blocks load their lines before they wait for the
// choice, which hides the probe (2 x 8 of 305 us of a 256^3 scan); the others find
// it made.
constexpr unsigned kFirstBlocks = 152 * 4;

__device__ __forceinline__ bool left_to_envelope(const int *wide)
{
    cudaGridDependencySynchronize();
    return wide && *(const volatile int *)wide;
}

// A launch that need not wait for the end of the probe before it.
template <class... Args, class... Given>
cudaError_t launch_after_probe(void (*kernel)(Args...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                               Given... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Args>(args)...);
}

// The outward scan (edt_scan.cu), lines of at most kScanMaxLine voxels; vcap:
// values above it only matter as "above it".  Line flags: the ends depend on
// imported hulls; the whole line is left to the float envelope.  wide (device,
// null: never): set by the probe when the envelope is to take every line, and
// the scan then does nothing.
constexpr int kScanEnds = 1, kScanWhole = 2;
int launch_pore_probe(const float *fin, const Lines &Ls, float res, float vcap, int periodic, int *wide,
                      const int **choice, cudaStream_t st);
int launch_scan(const float *fin, float *fout, const Lines &Ls, float res, const pmg_axis_cfg &cfg, int form,
                const MorphEpi &me, float vcap, uint8_t *flag, const int *wide, cudaStream_t st);
// flag_buf (optional): flag_cap ints for the per-line flags; without it they
// come from the stream-ordered scratch pool.
int launch_envelope(const float *fin, float *fout, const Lines &Ls, float res,
                    const pmg_axis_cfg &cfg, int num_hull, int form, const MorphEpi &me,
                    cudaStream_t st, int cap = INT_MAX, int *flag_buf = nullptr, long long flag_cap = 0,
                    float vcap = INFINITY);
int edt3d_run(const uint8_t *img, float *out, float *tmp, const int64_t *shape, const float *res,
              const pmg_axis_cfg *cfg, int num_hull, int form, cudaStream_t st, int *flag_buf = nullptr,
              long long flag_cap = 0);

} // namespace pmg
