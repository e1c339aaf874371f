// Exact Euclidean distance transform on GB300 (sm_103a).
//
// A transform is a linear pass along axis 0 and two envelope passes; edt3d_run
// gives each the first of these that takes its sizes:
//
//  * the linear pass: k_lin (edt_lattice.cu), counts for a lattice pass behind
//    it or squared distances; k_pass0 here for periodic lines of voxel sizes that
//    are no power of two and for lines beyond 2048;
//  * an envelope pass of power-of-two voxels, lines of at most 1024: the integer
//    lattice (edt_lattice.cu);
//  * an envelope pass of other voxel sizes, or of a voxel size that is larger than
//    an earlier axis's (or less than 2^-16 of it), lines of at most 1024: the
//    outward scan (edt_scan.cu), or the float envelope where a probe finds its
//    pores wide;
//  * longer lines: the exact integer stream (edt_exact.cu) where the sizes allow
//    it, the float envelope otherwise.
//
// Lines that the lattice and the scan cannot finish are handed back to the float
// envelope here: whole (k_envelope_whole), or their periodic ends alone
// (k_lattice_ends, k_envelope_ends).  The float kernels run one thread per 1-D
// line, lanes of a warp on neighbouring lines so that the strided axes are read
// and written coalesced:
//
//  * k_pass0     -- the linear two-sweep pass of squared_edt_1d
//                   (src/pmmoto/filters/distance/_distance.hpp:135-182) with
//                   the periodic correctors of _distance.pyx:240-279 /
//                   euclidean_distance_transform.py:395-447 found in-kernel.
//  * k_envelope  -- the lower envelope of parabolas of
//                   squared_edt_1d_parabolic (_distance.hpp:184-272) with the
//                   periodic boundary hulls of return_boundary_hull
//                   (_distance.hpp:296-356) computed in-kernel from the same
//                   line, so the MPI feature exchange of the reference becomes
//                   index arithmetic.
//
// The envelope stack is kept as a bitmask of surviving vertices in shared
// memory (one bit per voxel of the line, words interleaved across the block so
// every access is bank-conflict free).  A vertex's height is re-read from the
// input line and a segment's range is recomputed from the two neighbouring
// vertices with the same float expression the reference used when it pushed
// the segment, so the result is bit-identical while the per-line state is
// n/8 bytes instead of 16 n bytes.
//
// All floating-point steps use round-to-nearest intrinsics with no
// multiply-add contraction, in the reference's operation order.
#include <cfloat>
#include <cmath>
#include <algorithm>

#include "edt_internal.cuh"

namespace pmg {

// ---------------------------------------------------------------------------
// pass 0: squared_edt_1d along axis `ax`
// ---------------------------------------------------------------------------
__global__ void k_pass0(const uint8_t *__restrict__ img, float *__restrict__ out, Lines Ls,
                        float res, pmg_axis_cfg cfg)
{
    const long long nlines = Ls.count();
    for (long long li = blockIdx.x * (long long)blockDim.x + threadIdx.x; li < nlines;
         li += (long long)gridDim.x * blockDim.x) {
        const LineGeo g = line_addr(Ls, li);
        const uint8_t *in = img + g.base;
        float *d = out + g.base;
        const long long st = g.stride;
        const int n = g.n;
        float lc = INFINITY, uc = INFINITY;
        if (cfg.periodic) {
            int F = -1, L = -1;
            for (int i = cfg.f_lo; i < n; i++)
                if (in[i * st] == 0) {
                    F = i;
                    break;
                }
            for (int i = n - cfg.l_hi - 1; i >= cfg.l_lo; i--)
                if (in[i * st] == 0) {
                    L = i;
                    break;
                }
            if (F != -1)
                uc = (float)(F + cfg.a_u);
            if (L != -1)
                lc = (float)(n - L + cfg.a_l);
        }
        // forward sweep (reset at zeros, restart at a change of nonzero value)
        uint8_t seg = in[0];
        float prev = seg == 0 ? 0.0f : fmul(lc, res);
        d[0] = prev;
        uint8_t prev_v = seg;
        for (int i = 1; i < n; i++) {
            const uint8_t v = in[i * st];
            float cur;
            if (v == 0) {
                cur = 0.0f;
            } else if (v == seg) {
                cur = fadd(prev, res);
            } else {
                cur = res;
                d[(i - 1) * st] = prev_v != 0 ? res : 0.0f;
                seg = v;
            }
            d[i * st] = cur;
            prev = cur;
            prev_v = v;
        }
        // clamp the last voxel, backward sweep, square, inf -> FLT_MAX
        float b = d[(n - 1) * st];
        const float ucr = fmul(uc, res);
        if (b > ucr)
            b = ucr;
        {
            float q = fmul(b, b);
            d[(n - 1) * st] = q == INFINITY ? FLT_MAX : q;
        }
        for (int i = n - 2; i >= 0; i--) {
            const float a = d[i * st];
            b = fminf(a, fadd(b, res));
            const float q = fmul(b, b);
            d[i * st] = q == INFINITY ? FLT_MAX : q;
        }
    }
}

// ---------------------------------------------------------------------------
// envelope stack kept as a bitmask in shared memory
// ---------------------------------------------------------------------------
struct Entry {
    int v;
    float h;
};

struct Stack {
    uint32_t *bm; // word w of this thread at bm[w * nthr]
    int nthr;
    // imported lower hulls, bottom -> top (given ranges)
    int lv[kMaxHull];
    float lh[kMaxHull], lr[kMaxHull];
    int nl;
    // imported upper hulls pushed after the native vertices
    int uv[kMaxHull];
    float uh[kMaxHull], ur[kMaxHull];
    int nu;
    // native vertices (bits); ntv = topmost native vertex or -1
    int nn, ntv;
    // cached top of the whole stack
    int tv;
    float th, tr;

    __device__ __forceinline__ uint32_t &word(int w) { return bm[(long long)w * nthr]; }
    __device__ __forceinline__ void setbit(int v) { word(v >> 5) |= (1u << (v & 31)); }
    __device__ __forceinline__ void clrbit(int v) { word(v >> 5) &= ~(1u << (v & 31)); }
    // highest set bit strictly below v (callers guarantee one exists; the
    // search still stops at word 0 so a broken invariant cannot leave the
    // thread's shared-memory words)
    __device__ __forceinline__ int prev_bit(int v)
    {
        int w = v >> 5;
        uint32_t m = word(w) & ((1u << (v & 31)) - 1u);
        while (m == 0) {
            if (w == 0)
                return 0;
            --w;
            m = word(w);
        }
        return (w << 5) + 31 - __clz(m);
    }
    // lowest set bit strictly above v, or -1 if none below `lim` bits
    __device__ __forceinline__ int next_bit(int v, int nwords)
    {
        int w = (v + 1) >> 5;
        if (w >= nwords)
            return -1;
        uint32_t m = (v + 1) & 31 ? word(w) & ~((1u << ((v + 1) & 31)) - 1u) : word(w);
        while (m == 0) {
            if (++w >= nwords)
                return -1;
            m = word(w);
        }
        return (w << 5) + __ffs(m) - 1;
    }
    __device__ __forceinline__ void clear(int nwords)
    {
        for (int w = 0; w < nwords; w++)
            word(w) = 0u;
    }
};

// Heights of a line by vertex: read from the line in global memory ...
struct LineGlobal {
    const float *p;
    long long st;
    __device__ __forceinline__ float operator()(int v) const { return p[v * st]; }
    __device__ __forceinline__ LineGlobal from(int v) const { return {p + v * st, st}; }
};

// ... or with both line ends staged in shared memory (the first and last
// kEndWin positions, slot v of this thread's line at s[v * sst]; global
// memory in between, as floats or as counts of voxels).
constexpr int kEndWin = 32;

template <class T>
struct LineEnds {
    const T *p;
    long long st;
    const float *s;
    int sst, n, off;
    float res;
    __device__ __forceinline__ float operator()(int v) const
    {
        v += off;
        if (v < kEndWin)
            return s[v * sst];
        if (v >= n - kEndWin)
            return s[(v - n + 2 * kEndWin) * sst];
        return height_of(p + v * st, res);
    }
    __device__ __forceinline__ LineEnds from(int v) const
    {
        LineEnds l = *this;
        l.off += v;
        return l;
    }
};

// Range of the native vertex `v` = intersection with the entry below it.
template <class L>
__device__ __forceinline__ float native_range(Stack &S, const L &line, int v, float h, float aniso,
                                              int below_native_count)
{
    if (below_native_count > 0) {
        int pv = S.prev_bit(v);
        return isect(h, (float)v, line(pv), (float)pv, aniso);
    }
    if (S.nl > 0)
        return isect(h, (float)v, S.lh[S.nl - 1], (float)S.lv[S.nl - 1], aniso);
    return -INFINITY;
}

// Pop the top entry and reload the cache with the new top.
template <class L>
__device__ __forceinline__ void pop_top(Stack &S, const L &line, float aniso)
{
    if (S.nu > 0) {
        --S.nu;
        if (S.nu > 0) {
            S.tv = S.uv[S.nu - 1];
            S.th = S.uh[S.nu - 1];
            S.tr = S.ur[S.nu - 1];
            return;
        }
    } else if (S.nn > 0) {
        S.clrbit(S.ntv);
        --S.nn;
        S.ntv = S.nn > 0 ? S.prev_bit(S.ntv) : -1;
    } else {
        --S.nl;
    }
    if (S.nn > 0) {
        S.tv = S.ntv;
        S.th = line(S.ntv);
        S.tr = native_range(S, line, S.ntv, S.th, aniso, S.nn - 1);
    } else {
        S.tv = S.lv[S.nl - 1];
        S.th = S.lh[S.nl - 1];
        S.tr = S.lr[S.nl - 1];
    }
}

// update_hull (_distance.hpp:89-112) for vertex i with height f; `kind`
// 0 = native vertex (a bit), 1 = imported upper hull.
template <class L>
__device__ __forceinline__ void insert(Stack &S, const L &line, int i, float f, float aniso, int kind)
{
    float s = isect(f, (float)i, S.th, (float)S.tv, aniso);
    while (S.nl + S.nn + S.nu > 1 && s <= S.tr) {
        pop_top(S, line, aniso);
        s = isect(f, (float)i, S.th, (float)S.tv, aniso);
    }
    if (kind == 0) {
        S.setbit(i);
        ++S.nn;
        S.ntv = i;
    } else {
        S.uv[S.nu] = i;
        S.uh[S.nu] = f;
        S.ur[S.nu] = s;
        ++S.nu;
    }
    S.tv = i;
    S.th = f;
    S.tr = s;
}

// Build the envelope of a line segment [0, n) of `line` with no imports:
// entry (0, f(0)) at the bottom, then vertices 1..n-1.
template <class L>
__device__ __forceinline__ void build_plain(Stack &S, const L &line, int n, float aniso)
{
    S.nl = 0;
    S.nu = 0;
    S.setbit(0);
    S.nn = 1;
    S.ntv = 0;
    S.tv = 0;
    S.th = line(0);
    S.tr = -INFINITY;
    for (int i = 1; i < n; i++)
        insert(S, line, i, line(i), aniso, 0);
}

// Iterator over the final stack, bottom to top.
struct Iter {
    int phase; // 0 lower, 1 native, 2 upper, 3 done
    int idx;   // lower/upper index or native vertex
};

template <class L>
__device__ __forceinline__ bool iter_next(Stack &S, Iter &it, const L &line, int nwords, Entry &e, int &is_lower,
                                          float &given_r)
{
    for (;;) {
        if (it.phase == 0) {
            if (it.idx < S.nl) {
                e.v = S.lv[it.idx];
                e.h = S.lh[it.idx];
                given_r = S.lr[it.idx];
                is_lower = 1;
                ++it.idx;
                return true;
            }
            it.phase = 1;
            it.idx = -1;
        }
        if (it.phase == 1) {
            int nb = S.nn > 0 ? S.next_bit(it.idx, nwords) : -1;
            if (nb >= 0) {
                it.idx = nb;
                e.v = nb;
                e.h = line(nb);
                is_lower = 0;
                return true;
            }
            it.phase = 2;
            it.idx = 0;
        }
        if (it.phase == 2) {
            if (it.idx < S.nu) {
                e.v = S.uv[it.idx];
                e.h = S.uh[it.idx];
                is_lower = 0;
                ++it.idx;
                return true;
            }
            it.phase = 3;
        }
        return false;
    }
}

// return_boundary_hull (_distance.hpp:296-356) on segment [start, start+nv)
// of the line: keep up to num_hull+1 finite parabolas from the chosen end,
// vertices and ranges shifted by `corr`.  Returns the count; the bitmask is
// left cleared.
template <class L>
__device__ int boundary_hull(Stack &S, const L &line, int start, int nv, float aniso, int num_hull, int corr,
                             bool forward, int *ov, float *oh, float *orr)
{
    const L seg = line.from(start);
    if (nv <= 0)
        return 0;
    if (nv == 1) {
        const float f0 = seg(0);
        if (f0 < FLT_MAX) {
            ov[0] = corr;
            oh[0] = f0;
            orr[0] = INFINITY;
            return 1;
        }
        // the reference reads its "phantom" second slot here: vertex 0, height 0
        ov[0] = corr;
        oh[0] = 0.0f;
        orr[0] = INFINITY;
        return 1;
    }
    const int nwords = (nv + 31) >> 5;
    build_plain(S, seg, nv, aniso);
    const int top = S.nn - 1; // stack index of the top entry
    const int keep = num_hull < top ? num_hull : top;
    int cnt = 0;
    if (forward) {
        int v = -1;
        float prev_h = 0.0f;
        int prev_v = 0;
        for (int k = 0; k <= top && cnt <= keep; k++) {
            v = S.next_bit(v, nwords);
            const float h = seg(v);
            const float r = k == 0 ? -INFINITY : isect(h, (float)v, prev_h, (float)prev_v, aniso);
            if (h < FLT_MAX) {
                ov[cnt] = v + corr;
                oh[cnt] = h;
                orr[cnt] = fadd(r, (float)corr);
                ++cnt;
                if (h == 0.9f)
                    break;
            }
            prev_h = h;
            prev_v = v;
        }
    } else {
        int v = S.ntv;
        float h = seg(v);
        for (int k = top; k >= 0 && cnt <= keep; k--) {
            int pv = 0;
            float ph = 0.0f, r;
            if (k > 0) {
                pv = S.prev_bit(v);
                ph = seg(pv);
                r = isect(h, (float)v, ph, (float)pv, aniso);
            } else {
                r = -INFINITY;
            }
            if (h < FLT_MAX) {
                ov[cnt] = v + corr;
                oh[cnt] = h;
                orr[cnt] = fadd(r, (float)corr);
                ++cnt;
                if (h == 0.9f)
                    break;
            }
            v = pv;
            h = ph;
        }
    }
    S.clear(nwords);
    return cnt;
}

// ---------------------------------------------------------------------------
// envelope pass along axis `ax`: fin -> fout (out of place)
// ---------------------------------------------------------------------------

// The imported boundary hulls of a periodic line (return_boundary_hull on the
// segment before the first zero and after the last zero, the far end's hull
// becoming the lower imports).  A zero height is exactly a zero voxel of the
// original image: pass 0 gives 0 only there and every later pass keeps it, all
// other values being >= res^2 > 0.

// near end (forward) -> upper imports
template <class L>
__device__ __forceinline__ void load_upper(Stack &S, const L &line, int n, float aniso, const pmg_axis_cfg &cfg,
                                           int num_hull, int *up_v, float *up_h, float *up_r, int &n_up)
{
    int bf = -1;
    for (int i = cfg.hf_lo; i < n; i++)
        if (line(i) == 0.0f) {
            bf = i;
            break;
        }
    const int nv = bf == -1 ? n - cfg.hf_lo : bf - cfg.hf_lo + 1;
    n_up = boundary_hull(S, line, cfg.hf_lo, nv, aniso, num_hull, 0, true, up_v, up_h, up_r);
}

// far end (backward) -> lower imports into S, given in top-down order
template <class L>
__device__ __forceinline__ void load_lower(Stack &S, const L &line, int n, float aniso, const pmg_axis_cfg &cfg,
                                           int num_hull)
{
    int bb = -1;
    for (int i = n - cfg.hb_hi - 1; i >= 0; i--)
        if (line(i) == 0.0f) {
            bb = i;
            break;
        }
    int lo_v[kMaxHull];
    float lo_h[kMaxHull], lo_r[kMaxHull];
    const int start = bb == -1 ? 0 : bb, nv = n - start - cfg.hb_hi;
    const int n_lo = boundary_hull(S, line, start, nv, aniso, num_hull, -nv, false, lo_v, lo_h, lo_r);
    // the reference pushes the lower list in reverse (rbegin..rend)
    for (int j = 0; j < n_lo; j++) {
        S.lv[j] = lo_v[n_lo - 1 - j];
        S.lh[j] = lo_h[n_lo - 1 - j];
        S.lr[j] = lo_r[n_lo - 1 - j];
    }
    S.nl = n_lo;
}

template <class L>
__device__ __forceinline__ void load_imports(Stack &S, const L &line, int n, float aniso, const pmg_axis_cfg &cfg,
                                             int num_hull, int *up_v, float *up_h, float *up_r, int &n_up)
{
    load_upper(S, line, n, aniso, cfg, num_hull, up_v, up_h, up_r, n_up);
    load_lower(S, line, n, aniso, cfg, num_hull);
}

// Evaluation sweep over the final stack (bottom to top), written for
// positions [i_lo, i_hi) of the line.
template <class L>
__device__ __forceinline__ void evaluate(Stack &S, const L &line, int nwords, float aniso, int form,
                                         const MorphEpi &me, const LineGeo &g, float *o, int i_lo, int i_hi)
{
    Iter it{0, 0};
    Entry cur, nxt;
    int is_lower;
    float given_r;
    iter_next(S, it, line, nwords, cur, is_lower, given_r);
    bool has_next = iter_next(S, it, line, nwords, nxt, is_lower, given_r);
    float nr = has_next ? (is_lower ? given_r : isect(nxt.h, (float)nxt.v, cur.h, (float)cur.v, aniso)) : INFINITY;
    for (int i = i_lo; i < i_hi; i++) {
        const float fi = (float)i;
        while (nr < fi) {
            cur = nxt;
            has_next = iter_next(S, it, line, nwords, nxt, is_lower, given_r);
            nr = has_next ? (is_lower ? given_r : isect(nxt.h, (float)nxt.v, cur.h, (float)cur.v, aniso))
                          : INFINITY;
        }
        const float dx = (float)(i - cur.v);
        float val = fadd(fmul(aniso, fmul(dx, dx)), cur.h);
        if (form == PMG_EDT_MORPH) {
            morph_store(me, g, i, val);
            continue;
        }
        if (form == PMG_EDT_DIST)
            val = __fsqrt_rn(val);
        o[i * g.stride] = val;
    }
}

// The stack before the natives: the lower imports, or native 0; the first native
// to push.
template <class L>
__device__ __forceinline__ int stack_base(Stack &S, const L &line)
{
    if (S.nl > 0) {
        S.nn = 0;
        S.ntv = -1;
        S.tv = S.lv[S.nl - 1];
        S.th = S.lh[S.nl - 1];
        S.tr = S.lr[S.nl - 1];
        return 0;
    }
    S.setbit(0);
    S.nn = 1;
    S.ntv = 0;
    S.tv = 0;
    S.th = line(0);
    S.tr = -INFINITY;
    return 1;
}

// The reference's envelope of a whole line.
template <class L>
__device__ __forceinline__ void envelope_line(Stack &S, const L &line, const LineGeo &g, float aniso,
                                              const pmg_axis_cfg &cfg, int num_hull, int form, const MorphEpi &me,
                                              float *fout)
{
    const int n = g.n;
    const int nwords = (n + 31) >> 5;
    S.clear(nwords);
    S.nl = 0;
    S.nu = 0;
    int up_v[kMaxHull];
    float up_h[kMaxHull], up_r[kMaxHull];
    int n_up = 0;
    if (cfg.periodic)
        load_imports(S, line, n, aniso, cfg, num_hull, up_v, up_h, up_r, n_up);
    for (int i = stack_base(S, line); i < n; i++)
        insert(S, line, i, line(i), aniso, 0);
    for (int j = 0; j < n_up; j++)
        insert(S, line, up_v[j] + n, up_h[j], aniso, 1);
    evaluate(S, line, nwords, aniso, form, me, g, fout + g.base, 0, n);
}

__global__ void k_envelope(const float *__restrict__ fin, float *__restrict__ fout, Lines Ls, float res,
                           pmg_axis_cfg cfg, int num_hull, int form, MorphEpi me, int redo)
{
    const long long nlines = Ls.count();
    extern __shared__ uint32_t smem_bm[];
    const float aniso = fmul(res, res);
    Stack S;
    S.bm = smem_bm + threadIdx.x;
    S.nthr = blockDim.x;
    for (long long li = blockIdx.x * (long long)blockDim.x + threadIdx.x; li < nlines;
         li += (long long)gridDim.x * blockDim.x) {
        const LineGeo g = line_addr(Ls, li);
        // second chance for lines the exact streaming kernel handed back
        if (redo && !line_marked(fout, me, g, form))
            continue;
        envelope_line(S, LineGlobal{fin + g.base, g.stride}, g, aniso, cfg, num_hull, form, me, fout);
    }
}

// Lines that a scan or a lattice pass left to the envelope, or (wide) all of them.
template <class T>
struct LineOf {
    const T *p;
    long long st;
    float res;
    __device__ __forceinline__ float operator()(int v) const { return height_of(p + v * st, res); }
    __device__ __forceinline__ LineOf from(int v) const { return {p + v * st, st, res}; }
};

// A solid on the line at all (a lattice pass flags every line with a voxel out of
// its range, a probe leaves all lines).
template <class L>
__device__ __forceinline__ bool some_height(const L &line, int n)
{
    bool some = false;
    for (int i = 0; i < n && !some; i += 16) {
#pragma unroll
        for (int u = 0; u < 16; u++)
            some |= i + u < n && line(min(i + u, n - 1)) < FLT_MAX;
    }
    return some;
}

__device__ __forceinline__ bool whole_flag(uint8_t f) { return f & kScanWhole; }
__device__ __forceinline__ bool whole_flag(uint16_t f) { return (f & 0xff) == kWholeLine; }

template <class T, class F>
__global__ void k_envelope_whole(const T *__restrict__ fin, float *__restrict__ fout, Lines Ls, float res, float resh,
                                 pmg_axis_cfg cfg, int num_hull, int form, MorphEpi me, const F *__restrict__ flag,
                                 const int *__restrict__ wide)
{
    const bool all = wide && *wide;
    if (!all && !flag)
        return;
    const long long nlines = Ls.count();
    extern __shared__ uint32_t smem_bm[];
    const float aniso = fmul(res, res);
    Stack S;
    S.bm = smem_bm + threadIdx.x;
    S.nthr = blockDim.x;
    const float none = form == PMG_EDT_DIST ? __fsqrt_rn(FLT_MAX) : FLT_MAX;
    const int lane = threadIdx.x & 31;
    for (long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; first < nlines;
         first += (long long)gridDim.x * blockDim.x) {
        const long long li = first + lane;
        const bool mine = li < nlines && (all || whole_flag(flag[li]));
        const LineGeo g = line_addr(Ls, mine ? li : first);
        bool empty = false;
        if (mine) {
            const LineOf<T> line{fin + g.base, g.stride, resh};
            // (a scan flags no line without a height; one pass of an empty 1000 x 1000
            // image: 0.77 ms without this look at a line, 0.07 with it)
            empty = form != PMG_EDT_MORPH && (all || sizeof(F) != 1) &&
                    !(cfg.periodic && (g.n - cfg.hf_lo < 2 || g.n - cfg.hb_hi < 2)) && !some_height(line, g.n);
            if (!empty)
                envelope_line(S, line, g, aniso, cfg, num_hull, form, me, fout);
        }
        if (g.stride != 1) {
            if (empty) {
#pragma unroll 8
                for (int i = 0; i < g.n; i++)
                    fout[g.base + i * g.stride] = none;
            }
            continue;
        }
        // (rows: the warp writes one after the other)
        for (unsigned e = __ballot_sync(0xffffffffu, empty); e; e &= e - 1) {
            const long long at = __shfl_sync(0xffffffffu, g.base, __ffs(e) - 1);
            for (int i = lane; i < g.n; i += 32)
                fout[at + i] = none;
        }
    }
}

// ---------------------------------------------------------------------------
// flagged lines
// ---------------------------------------------------------------------------
// Lines the lattice and scan passes flag (edt_lattice.cu, edt_scan.cu) depend
// on the imported hulls at their ends, or need the reference's float envelope
// as a whole.

// One line replayed with the float envelope: a line without a zero height as a
// whole, any other by its end segments only -- the lower imports with
// the voxels up to the first zero, and the voxels from the last zero with the
// upper imports.  No parabola can pop a zero off the stack, so these partial
// stacks and sweeps make the same float decisions as the whole line's.
// part: 3 for both ends, 1 for the low end or the whole line, 2 for the high end
// (nothing where the whole line is replayed), so that two threads can share a
// line.  bm: this thread's envelope bits, nthr threads apart.
template <class L>
__device__ __noinline__ void replay_line(uint32_t *bm, int nthr, const L &line, const LineGeo &g, float aniso,
                                         const pmg_axis_cfg &cfg, int num_hull, int form, const MorphEpi &me,
                                         float *fout, int part = 3)
{
    Stack S;
    S.bm = bm;
    S.nthr = nthr;
    const int n = g.n;
    const int nwords = (n + 31) >> 5;
    int z1 = -1, z2 = -1;
    for (int i = 0; i < n; i++)
        if (line(i) == 0.0f) {
            z1 = i;
            break;
        }
    for (int i = n - 1; i >= 0; i--)
        if (line(i) == 0.0f) {
            z2 = i;
            break;
        }
    S.clear(nwords);
    S.nl = 0;
    S.nu = 0;
    int up_v[kMaxHull];
    float up_h[kMaxHull], up_r[kMaxHull];
    int n_up = 0;
    const bool whole = z1 < 0;
    if (whole && part == 2)
        return;
    if (cfg.periodic && (whole || (part & 2)))
        load_upper(S, line, n, aniso, cfg, num_hull, up_v, up_h, up_r, n_up);
    if (cfg.periodic && (whole || (part & 1)))
        load_lower(S, line, n, aniso, cfg, num_hull);
    const int lo_end = whole ? n - 1 : z1; // last native of the lower stack
    // lower part: the imports below, natives up to lo_end
    if (whole || ((part & 1) && z1 > 0)) {
        for (int i = stack_base(S, line); i <= lo_end; i++)
            insert(S, line, i, line(i), aniso, 0);
        if (whole) {
            for (int j = 0; j < n_up; j++)
                insert(S, line, up_v[j] + n, up_h[j], aniso, 1);
            evaluate(S, line, nwords, aniso, form, me, g, fout + g.base, 0, n);
            return;
        }
        evaluate(S, line, nwords, aniso, form, me, g, fout + g.base, 0, z1);
        S.clear(nwords);
    }
    // upper part: the zero at z2 at the bottom, natives above it, the upper
    // imports on top
    if ((part & 2) && z2 < n - 1) {
        S.nl = 0;
        S.nu = 0;
        S.setbit(z2);
        S.nn = 1;
        S.ntv = z2;
        S.tv = z2;
        S.th = 0.0f;
        S.tr = -INFINITY;
        for (int i = z2 + 1; i < n; i++)
            insert(S, line, i, line(i), aniso, 0);
        for (int j = 0; j < n_up; j++)
            insert(S, line, up_v[j] + n, up_h[j], aniso, 1);
        evaluate(S, line, nwords, aniso, form, me, g, fout + g.base, z2 + 1, n);
    }
}

// The first and last kEndWin heights of 32 adjacent lines (l0, l0 + 1, ...; g:
// this lane's), staged by `parts` warps, this one being `part`.
template <class T>
__device__ __forceinline__ void stage_ends(float *se, const T *__restrict__ fin, const Lines &Ls, long long l0,
                                           int lines, const LineGeo &g, float res, int part, int parts)
{
    const int lane = threadIdx.x & 31, n = g.n;
    if (Ls.ax == 2) {
        // rows: lanes along the row, transposed on the way in
        const T *p0 = fin + line_addr(Ls, l0).base;
#pragma unroll 4
        for (int r = part; r < lines; r += parts) {
            const T *p = p0 + (long long)r * Ls.s2;
            const int u = n - kEndWin + lane;
            if (lane < n)
                se[lane * 33 + r] = height_of(p + lane, res);
            if (u >= 0)
                se[(kEndWin + lane) * 33 + r] = height_of(p + u, res);
        }
    } else {
        const T *p = fin + g.base;
#pragma unroll 8
        for (int v = part; v < kEndWin; v += parts) {
            const int u = n - kEndWin + v;
            if (v < n)
                se[v * 33 + lane] = height_of(p + v * g.stride, res);
            if (u >= 0)
                se[(kEndWin + v) * 33 + lane] = height_of(p + u * g.stride, res);
        }
    }
}

// Lines whose ends a scan flagged (kScanEnds alone: k_envelope_whole has the
// others), of any voxel size: a block takes `width` adjacent lines (unflagged ones
// idle), the lanes of warp 0 their low ends, or the line when it has no zero, and
// those of warp 1 their high ends, two chains that overlap.
// Both ends of the lines are staged in shared memory first, because the zero
// searches, hulls, pushes and the sweep read them again and again in dependent
// steps.
// Bound by the latency of those steps, and by the lanes of a warp popping
// different numbers of parabolas: with one lane for both ends a periodic 341 x
// 298 x 125 field took 0.80 ms here, now 0.57 ms.  A warp of 32 lines waits for
// the slowest at every push, so few lines are spread over more warps: eight
// to a warp where that leaves each scheduler a handful of warps at most.
constexpr int kEndBlock = 64;

__global__ void __launch_bounds__(kEndBlock) k_envelope_ends(const float *__restrict__ fin, float *__restrict__ fout,
                                                             Lines Ls, float res, pmg_axis_cfg cfg, int num_hull,
                                                             int form, MorphEpi me, const uint8_t *__restrict__ flag,
                                                             int width, const int *__restrict__ wide)
{
    if (wide && *wide)
        return;
    extern __shared__ uint32_t smem_bm[];
    __shared__ float s_ends[2 * kEndWin * 33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // tiles of lines that are adjacent in memory (along the second axis)
    const int tiles = (Ls.nb2 + width - 1) / width;
    const long long ntiles = (long long)Ls.nb1 * tiles;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int ra = (int)(t / tiles), kb = (int)(t - (long long)ra * tiles) * width;
        const int lines = min(width, Ls.nb2 - kb);
        const long long l0 = (long long)ra * Ls.nb2 + kb;
        const bool ends = lane < lines && flag[l0 + lane] == kScanEnds;
        if (!__any_sync(0xffffffffu, ends)) // the same for both warps
            continue;
        const LineGeo g = line_addr(Ls, l0 + min(lane, lines - 1));
        __syncthreads(); // (the previous tile's readers)
        stage_ends(s_ends, fin, Ls, l0, lines, g, res, w, 2);
        __syncthreads();
        if (!ends)
            continue;
        const LineEnds<float> line{fin + g.base, g.stride, s_ends + lane, 33, g.n, 0, res};
        replay_line(smem_bm + threadIdx.x, kEndBlock, line, g, fmul(res, res), cfg, num_hull, form, me, fout, 1 << w);
    }
}

// Flagged lines of the lattice passes (line_reach: how many positions from the
// low and the high end, or the whole line).  Heights are integer multiples K
// of res^2, so a voxel there is the smaller of the value the pass left and the
// imported parabolas, and only the imports have to be found: the last (first)
// num_hull + 1 finite entries of the hull of the far (near) segment.  They
// are wrapped one by one from the line's end -- the entry next to e is the
// vertex whose intersection with e lies closest, of equal ones the farthest
// (the reference pops on equality) -- by cross-multiplied integer
// comparisons, up to the zero that ends the segment or the distance from
// which no height could bring an intersection closer.  The reference compares
// rounded quotients: a best one within their rounding of another leaves the
// line to the float replay, and so do lines flagged as a whole and searches
// too long for 32-bit products.  A block takes 32 adjacent lines, warp 0
// their low ends and warp 1 their high ones, so that the two independent
// chains overlap.
// Bound by the latency of those chains.  Building the reference's hull stacks
// instead kept a warp in divergent pops and divisions: 1024^3 field 1.8 ms
// over both passes, 128^3 pack 0.54 ms.
constexpr int kWrapMax = 255;        // farthest entry
constexpr float kTall = 2097152.0f;  // tallest height (their products' differences stay below 2^31)

template <class T>
__global__ void __launch_bounds__(64) k_lattice_ends(const T *__restrict__ fin, float *__restrict__ fout, Lines Ls,
                                                     float res, float resh, pmg_axis_cfg cfg, int num_hull, int form,
                                                     uint16_t *__restrict__ flag, int defer)
{
    extern __shared__ uint32_t smem_bm[]; // envelope bits of the replays: [nwords][32]
    __shared__ float s_ends[2 * kEndWin * 33];
    __shared__ int s_hard[32];
    const float aniso = fmul(res, res), inv_a = 1.0f / aniso;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int tiles = (Ls.nb2 + 31) / 32;
    const long long ntiles = (long long)Ls.nb1 * tiles;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int ra = (int)(t / tiles), kb = (int)(t - (long long)ra * tiles) * 32;
        const int lines = min(32, Ls.nb2 - kb);
        const long long l0 = (long long)ra * Ls.nb2 + kb;
        const int all = lane < lines ? flag[l0 + lane] : 0, fl = whole_flag((uint16_t)all) ? 0 : all;
        if (!__any_sync(0xffffffffu, fl)) // the same for both warps
            continue;
        const LineGeo g = line_addr(Ls, l0 + min(lane, lines - 1));
        const int n = g.n;
        __syncthreads(); // (the previous tile's readers)
        if (w == 0)
            s_hard[lane] = 0;
        stage_ends(s_ends, fin, Ls, l0, lines, g, resh, w, 2);
        __syncthreads();
        const LineEnds<T> line{fin + g.base, g.stride, s_ends + lane, 33, n, 0, resh};
        const int reach = w == 0 ? fl & 0xff : fl >> 8;
        if (reach > 0) {
            // positions of the segment from its end that faces the line
            const int p0 = w == 0 ? n - cfg.hb_hi - 1 : cfg.hf_lo, dir = w == 0 ? -1 : 1;
            const int most = w == 0 ? n - cfg.hb_hi : n - cfg.hf_lo;
            // (a segment of one voxel without a solid one: the reference's phantom import)
            bool hard = most < 2, far = false; // far: out of this search's range
            // entries (position q, height K); q = -1: none
            int eq[kMaxHull], ek[kMaxHull];
#pragma unroll
            for (int c = 0; c < kMaxHull; c++) {
                eq[c] = -1;
                ek[c] = 0;
            }
            if (!hard) {
                // (a height beyond kTall leaves the line to the float replay: 32-bit products)
                auto height = [&](int q) -> int {
                    const float f = line(p0 + dir * q), k = fmul(f, inv_a);
                    far = far || (f < FLT_MAX && k > kTall);
                    return f >= FLT_MAX || k > kTall ? -1 : (int)k;
                };
                int e = 0, ke = height(0);
                while (ke < 0 && ++e < most)
                    ke = height(e);
                if (e < most) {
                    eq[0] = e;
                    ek[0] = ke;
                }
#pragma unroll
                for (int c = 1; c < kMaxHull; c++) {
                    if (c > num_hull || e >= most || ke == 0)
                        continue; // (a zero ends the segment)
                    // distance from e of the intersection with q: N / (2 D), smallest
                    int b = most, kb2 = 0, nb = 0, db = 1;
                    bool near = false; // another one within the rounding of the best
                    for (int q = e + 1; q < most; q++) {
                        const int d = q - e;
                        // no height from here on comes within 1 / 2 of the best
                        if (b < most && (d * d - ke) * db - nb * d > d * db)
                            break;
                        if (d > kWrapMax) {
                            far = true;
                            break;
                        }
                        const int k = height(q);
                        if (k < 0)
                            continue;
                        const int N = k - ke + d * d;
                        const int diff = N * db - nb * d;
                        const float tol =
                            2.4e-7f * (float)(2 * max(k, max(ke, kb2)) + 6 * (q + 1)) * (float)(d * db);
                        if (b < most && diff != 0 && (float)abs(diff) < tol)
                            near = true;
                        else if (b == most || diff < 0)
                            near = false;
                        if (b == most || diff <= 0) {
                            b = q;
                            kb2 = k;
                            nb = N;
                            db = d;
                        }
                        if (k == 0)
                            break;
                    }
                    hard = hard || near;
                    e = b;
                    ke = kb2;
                    if (e < most) {
                        eq[c] = e;
                        ek[c] = ke;
                    }
                }
            }
            if (far || hard) {
                atomicMax(&s_hard[lane], far ? 2 : 1);
            } else {
                // import c lies eq[c] + 1 beyond the line's end
                float *o = fout + g.base + (w == 0 ? 0 : n - 1) * g.stride;
                const long long step = w == 0 ? g.stride : -g.stride;
                for (int i0 = 0; i0 < reach; i0 += 4) {
                    float cur[4];
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        cur[u] = i0 + u < reach ? o[(i0 + u) * step] : 0.0f;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int i = i0 + u;
                        int best = 1 << 30;
#pragma unroll
                        for (int c = 0; c < kMaxHull; c++)
                            if (eq[c] >= 0) {
                                const int d = i + 1 + eq[c];
                                best = min(best, ek[c] + d * d);
                            }
                        float val = best < 1 << 30 ? fmul((float)best, aniso) : FLT_MAX;
                        if (form == PMG_EDT_DIST)
                            val = __fsqrt_rn(val);
                        // (the two ends may reach the same voxel; values are >= 0)
                        if (val < cur[u])
                            atomicMin(reinterpret_cast<int *>(o + i * step), __float_as_int(val));
                    }
                }
            }
        }
        __syncthreads();
        if (w > 0)
            continue;
        // many such lines: as a whole, by the kernel that follows
        const int hard = s_hard[lane];
        const bool many = defer && __popc(__ballot_sync(0xffffffffu, hard == 2)) >= 16;
        if (many && hard == 2)
            flag[l0 + lane] = kWholeLine;
        else if (hard)
            replay_line(smem_bm + lane, 32, line, g, aniso, cfg, num_hull, form, MorphEpi{}, fout);
    }
}

template <class T>
int launch_lattice_ends(const T *fin, float *fout, const Lines &Ls, float res, float res_height, const pmg_axis_cfg &cfg,
                        int num_hull, int form, uint16_t *flag, int defer, cudaStream_t st)
{
    const int n = (int)(Ls.ax == 0 ? Ls.s0 : Ls.ax == 1 ? Ls.s1 : Ls.s2);
    const size_t smem = (size_t)((n + 31) / 32) * 32 * 4;
    const long long tiles = (long long)Ls.nb1 * ((Ls.nb2 + 31) / 32);
    const int ps__ = prof_begin("k_lattice_ends", st);
    k_lattice_ends<T><<<grid_for(tiles, 1, 152LL * 64), 64, smem, st>>>(fin, fout, Ls, res, res_height, cfg, num_hull, form,
                                                                          flag, defer);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

template int launch_lattice_ends(const float *, float *, const Lines &, float, float, const pmg_axis_cfg &, int, int,
                                 uint16_t *, int, cudaStream_t);
template int launch_lattice_ends(const uint16_t *, float *, const Lines &, float, float, const pmg_axis_cfg &, int, int,
                                 uint16_t *, int, cudaStream_t);

int launch_ends_float(const float *fin, float *fout, const Lines &Ls, float res, const pmg_axis_cfg &cfg,
                      int num_hull, int form, const MorphEpi &me, const uint8_t *flag, const int *wide, cudaStream_t st)
{
    const int n = (int)(Ls.ax == 0 ? Ls.s0 : Ls.ax == 1 ? Ls.s1 : Ls.s2);
    const size_t smem = (size_t)((n + 31) / 32) * kEndBlock * 4;
    const int width = (long long)Ls.nb1 * ((Ls.nb2 + 31) / 32) * 2 <= 152LL * 4 * 4 ? 8 : 32;
    const long long tiles = (long long)Ls.nb1 * ((Ls.nb2 + width - 1) / width);
    const int ps__ = prof_begin("k_envelope_ends", st);
    k_envelope_ends<<<grid_for(tiles, 1, 152LL * 64), kEndBlock, smem, st>>>(
        fin, fout, Ls, res, cfg, num_hull, form, me, flag, width, wide);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
int launch_pass0(const uint8_t *img, float *out, const Lines &Ls, float res,
                 const pmg_axis_cfg &cfg, cudaStream_t st)
{
    const int block = 256;
    {
        const int ps__ = prof_begin("k_pass0", st);
        k_pass0<<<grid_for(Ls.count(), block, 1LL << 30), block, 0, st>>>(img, out, Ls, res, cfg);
        prof_end(ps__, (double)Ls.count() * (Ls.ax == 0 ? Ls.s0 : Ls.ax == 1 ? Ls.s1 : Ls.s2) * 5, st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

static int envelope_block(int n)
{
    // shared bitmask: ceil(n/32) words per thread; keep <= 48 KB per block
    int words = (n + 31) / 32;
    int block = 256;
    while (block > 32 && (size_t)words * block * 4 > 48 * 1024)
        block >>= 1;
    return block;
}

template <class T, class F>
int launch_whole(const T *fin, float *fout, const Lines &Ls, float res, float res_height, const pmg_axis_cfg &cfg,
                 int num_hull, int form, const MorphEpi &me, const F *flag, const int *wide, cudaStream_t st)
{
    const int n = (int)(Ls.ax == 0 ? Ls.s0 : Ls.ax == 1 ? Ls.s1 : Ls.s2), block = envelope_block(n);
    const size_t smem = (size_t)((n + 31) / 32) * block * 4; // (48 KB at most)
    const int ps__ = prof_begin("k_envelope_whole", st);
    k_envelope_whole<<<grid_for(Ls.count(), block, 1LL << 30), block, smem, st>>>(fin, fout, Ls, res, res_height, cfg, num_hull,
                                                                                 form, me, flag, wide);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

template int launch_whole(const float *, float *, const Lines &, float, float, const pmg_axis_cfg &, int, int,
                          const MorphEpi &, const uint16_t *, const int *, cudaStream_t);
template int launch_whole(const uint16_t *, float *, const Lines &, float, float, const pmg_axis_cfg &, int, int,
                          const MorphEpi &, const uint16_t *, const int *, cudaStream_t);

// power-of-two voxel size and lines of at most 1024 voxels (imported hull
// vertices then stay within the exact float range of the reference's
// intersection arithmetic)
bool window_path_ok(float res, int n)
{
    if (n > kScanMaxLine || !(res > 0.0f))
        return false;
    int ex = 0;
    const float m = frexpf(res, &ex);
    return m == 0.5f && ex > -40 && ex < 40;
}

int launch_envelope(const float *fin, float *fout, const Lines &Ls, float res,
                    const pmg_axis_cfg &cfg, int num_hull, int form, const MorphEpi &me,
                    cudaStream_t st, int cap, int *flag_buf, long long flag_cap, float vcap)
{
    const int n = (int)(Ls.ax == 0 ? Ls.s0 : Ls.ax == 1 ? Ls.s1 : Ls.s2);
    int block = envelope_block(n);
    size_t smem = (size_t)((n + 31) / 32) * block * 4;
    if (smem > 48 * 1024) // (lines far beyond a scan's)
        PMG_CUDA(cudaFuncSetAttribute(k_envelope, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    const int path = tune_value(kTuneEdtPath);
    // The outward scan, the float envelope on the lines that it hands over (wide
    // pores, unresolved near-ties), and their ends replayed on periodic lines.
    // A caller's flag buffer that does not hold one byte per line (lines of a few
    // voxels) leaves the pass to the float envelope, and so do periodic lines of
    // voxel sizes that are no power of two, whose near-ties are many (400 x 300 x
    // 300 pack, voxels of 2.25: 6.4 ms, the envelope 4.0 ms).
    const long long nl = Ls.count();
    const size_t flag_bytes = ((size_t)nl + 3) / 4 * 4; // (then the probe's choice)
    if (path == 0 && n <= kScanMaxLine && (!cfg.periodic || window_path_ok(res, n)) &&
        (!flag_buf || flag_bytes + sizeof(int) <= (size_t)flag_cap * sizeof(int))) {
        uint8_t *flag = (uint8_t *)flag_buf;
        if (!flag_buf)
            PMG_TRY(scratch_alloc((void **)&flag, flag_bytes + sizeof(int), st));
        const int *wide = nullptr;
        int s = launch_pore_probe(fin, Ls, res, vcap, cfg.periodic, (int *)(flag + flag_bytes), &wide, st);
        if (s == PMG_OK)
            s = launch_scan(fin, fout, Ls, res, cfg, form, me, vcap, flag, wide, st);
        if (s == PMG_OK && cfg.periodic)
            s = launch_ends_float(fin, fout, Ls, res, cfg, num_hull, form, me, flag, wide, st);
        if (s == PMG_OK)
            s = launch_whole(fin, fout, Ls, res, res, cfg, num_hull, form, me, flag, wide, st);
        const int s2 = flag_buf ? PMG_OK : scratch_free(flag, st);
        return s != PMG_OK ? s : s2;
    }
    int redo = 0;
    if (path != 2 && exact_path_ok(res, cfg, n)) {
        // exact integer streaming pass; lines it cannot finish are redone below
        PMG_TRY(launch_envelope_exact(fin, fout, Ls, res, form, me, st, cap));
        redo = 1;
    }
    {
        const int ps__ = prof_begin(redo ? "k_envelope_redo" : "k_envelope", st);
        k_envelope<<<grid_for(Ls.count(), block, redo ? 152LL * 8 : 1LL << 30), block, smem, st>>>(
            fin, fout, Ls, res, cfg, num_hull, form, me, redo);
        prof_end(ps__, redo ? 0.0 : (double)Ls.count() * n * 4 + (form == PMG_EDT_MORPH ? (double)Ls.count() * me.o2 : (double)Ls.count() * n * 4), st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

static int check_shape(const int64_t *shape, int nd)
{
    for (int d = 0; d < nd; d++) {
        if (shape[d] <= 0) {
            set_error("shape[%d] = %lld must be positive", d, (long long)shape[d]);
            return PMG_EINVAL;
        }
        if (shape[d] > PMG_MAX_LINE) {
            set_error("shape[%d] = %lld exceeds the line limit %d", d, (long long)shape[d],
                      PMG_MAX_LINE);
            return PMG_ERANGE;
        }
    }
    return PMG_OK;
}

// The linear pass of any voxel size: counts through the table of the running
// sums, except where periodic correctors start the sums elsewhere.
int launch_linear(const uint8_t *img, float *out, const int64_t *shape, float res, const pmg_axis_cfg &cfg,
                  cudaStream_t st)
{
    if (tune_value(kTuneEdtPath) == 0 && !cfg.periodic && lin_ok((int)shape[0], cfg))
        return launch_lin_float(img, out, shape, res, cfg, st);
    return launch_pass0(img, out, all_lines(shape, 0), res, cfg, st);
}

// EDT with one ping-pong buffer: pass 0 -> out, envelope 1: out -> tmp,
// envelope 2: tmp -> out.
int edt3d_run(const uint8_t *img, float *out, float *tmp, const int64_t *shape, const float *res,
              const pmg_axis_cfg *cfg, int num_hull, int form, cudaStream_t st, int *flag_buf,
              long long flag_cap)
{
    MorphEpi none{};
    LatticePlan P{};
    if (tune_value(kTuneEdtPath) == 0)
        P = lattice_plan(shape, res, cfg);
    // a 16-bit flag per line of the larger lattice pass
    const long long lines = (long long)shape[0] * std::max(P.cols ? shape[2] : 0, P.rows ? shape[1] : 0);
    if (flag_buf && lines > flag_cap * (long long)(sizeof(int) / sizeof(uint16_t)))
        P = LatticePlan{};
    uint16_t *flag = (uint16_t *)flag_buf;
    if (!flag_buf && (P.cols || P.rows))
        PMG_TRY(scratch_alloc((void **)&flag, sizeof(uint16_t) * (size_t)lines, st));
    int s = P.counts ? launch_lin_counts(img, (uint16_t *)out, shape, cfg[0], st)
                     : launch_linear(img, out, shape, res[0], cfg[0], st);
    if (s == PMG_OK)
        s = P.cols ? lattice_cols(P, out, tmp, shape, res, cfg, num_hull, flag, st)
                   : launch_envelope(out, tmp, all_lines(shape, 1), res[1], cfg[1], num_hull, PMG_EDT_SQUARED, none, st,
                                     INT_MAX, flag_buf, flag_cap);
    if (s == PMG_OK)
        s = P.rows ? lattice_rows(P, tmp, out, shape, res, cfg, num_hull, form, flag, st)
                   : launch_envelope(tmp, out, all_lines(shape, 2), res[2], cfg[2], num_hull, form, none, st, INT_MAX,
                                     flag_buf, flag_cap);
    const int s2 = flag_buf ? PMG_OK : scratch_free(flag, st);
    return s != PMG_OK ? s : s2;
}

} // namespace pmg

using namespace pmg;

extern "C" int pmg_edt3d(const uint8_t *img, float *out, const int64_t shape[3], const float res[3],
                         const pmg_axis_cfg cfg[3], int32_t num_hull, int32_t form, void *stream)
{
    if (!img || !out || !shape || !res || !cfg) {
        set_error("pmg_edt3d: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_shape(shape, 3));
    if (num_hull < 0 || num_hull + 1 > kMaxHull) {
        set_error("pmg_edt3d: num_hull %d outside [0, %d]", num_hull, kMaxHull - 1);
        return PMG_ERANGE;
    }
    cudaStream_t st = as_stream(stream);
    size_t bytes = (size_t)shape[0] * shape[1] * shape[2] * sizeof(float);
    void *tmp = nullptr;
    PMG_TRY(scratch_alloc(&tmp, bytes, st));
    int s = edt3d_run(img, out, (float *)tmp, shape, res, cfg, num_hull, form, st);
    int s2 = scratch_free(tmp, st);
    return s != PMG_OK ? s : s2;
}

extern "C" int pmg_edt2d(const uint8_t *img, float *out, const int64_t shape2[2], const float res[2],
                         const int32_t periodic[2], int32_t num_hull, int32_t form, void *stream)
{
    if (!img || !out || !shape2 || !res || !periodic) {
        set_error("pmg_edt2d: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_shape(shape2, 2));
    if (num_hull < 0 || num_hull + 1 > kMaxHull) {
        set_error("pmg_edt2d: num_hull %d outside [0, %d]", num_hull, kMaxHull - 1);
        return PMG_ERANGE;
    }
    cudaStream_t st = as_stream(stream);
    const int64_t shape[3] = {1, shape2[0], shape2[1]};
    pmg_axis_cfg c_lin = {periodic[1], 0, 0, 0, 1, 0, 0, 0};
    pmg_axis_cfg c_env = {periodic[0], 0, 0, 0, 1, 0, 0, 0};
    size_t bytes = (size_t)shape2[0] * shape2[1] * sizeof(float);
    void *tmp = nullptr;
    PMG_TRY(scratch_alloc(&tmp, bytes, st));
    MorphEpi none{};
    int s = launch_pass0(img, (float *)tmp, all_lines(shape, 2), res[1], c_lin, st);
    if (s == PMG_OK)
        s = launch_envelope((float *)tmp, out, all_lines(shape, 1), res[0], c_env, num_hull, form,
                            none, st);
    int s2 = scratch_free(tmp, st);
    return s != PMG_OK ? s : s2;
}
