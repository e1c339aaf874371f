// Distance transform of power-of-two voxels on an integer lattice (sm_103a), and
// the linear pass of every other voxel size.
//
// Where the voxel sizes are powers of two and a pass's own is the smallest of the
// axes so far, every height that it reads is K * res^2 with an integer K, and the
// reference's float passes return the exact minimum at every position where it is
// below kBig (edt_exact.cu has the rounding argument for heights below 2^24;
// taller ones meet such a parabola thousands of positions away, far beyond their
// rounding).  So the passes run on integers, pass by pass:
//
//  * k_lin       the linear pass (squared_edt_1d, _distance.hpp:135-182, with
//                the correctors of _distance.pyx:240-279): counts of voxels to
//                the nearest zero or restart, uint16, every position of a line
//                by its own segment of threads;
//  * k_par_cols  a strided envelope pass: min over v of K(v) + (x - v)^2, from
//                counts (K = count^2 times the squared ratio of the sizes) or
//                from heights;
//  * k_par_rows  the same along the contiguous axis, out to float32.
//
// min over |d| <= k of K(x + d) + d^2 is built one distance at a time as
//     g_k(x) = min(g_{k-1}(x), min(g_{k-1}(x - 1), g_{k-1}(x + 1)) + 2k - 1)
// (d^2 = 1 + 3 + ... + (2d - 1); a path that turns back costs more), with the
// line's heights in registers, two lines packed in the halves of 32-bit words.
// It stops as soon as every value of the block (warp) is at most (k + 1)^2,
// because a height farther away adds at least that much: the work follows
// the medium's own distances, with no window to choose beforehand.
//
// Periodic lines: a voxel whose minimum exceeds the squared distance to a
// line end may depend on the imported boundary hulls; that end of its line is
// flagged (k_lattice_ends).  Heights of kBig and more
// count as absent; a line left with such a value is flagged for the float
// envelope, unless no height of the volume can reach kBig.
#include <cfloat>
#include <algorithm>
#include <cmath>

#include "edt_internal.cuh"

namespace pmg {

// Packed 16-bit minima and maxima as single instructions (the vminu2 / vmaxu2
// intrinsics are sequences here: the 512 x 512 x 1024 field's row pass ran 115
// instructions per pair of voxels with them).
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Integers below 2^16 to and from float by the exponent of 2^23 (exact; the
// conversion instructions run at a fraction of the rate).
__device__ __forceinline__ float lo_float(uint32_t v) { return __uint_as_float(0x4B000000u | (v & 0xffffu)) - 8388608.0f; }
__device__ __forceinline__ float hi_float(uint32_t v) { return __uint_as_float(0x4B000000u | (v >> 16)) - 8388608.0f; }
__device__ __forceinline__ uint32_t pack_float2(float a, float b) // integers in [0, 2^16)
{
    return __byte_perm(__float_as_uint(a + 8388608.0f), __float_as_uint(b + 8388608.0f), 0x5410);
}

// ---------------------------------------------------------------------------
// linear pass
// ---------------------------------------------------------------------------
// "No zero so far": counts grow from here by at most the line length.
constexpr int kLinInf = 0x4000;
constexpr int kLinChunk = 8;       // positions a thread holds at once
constexpr int kLinChunks = 16;     // chunks per thread
constexpr int kLinWarps = 16;      // segments per line

struct LinTab {
    float v[kLinMaxLine + 1]; // squared distance of a count
};
struct NoTab {};
template <class OUT>
struct TabOf {
    using T = NoTab;
};
template <>
struct TabOf<float> {
    using T = LinTab;
};

// bytes != 0 -> 0x01 per byte
__device__ __forceinline__ uint32_t nz01(uint32_t v)
{
    return ((((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) >> 7) & 0x01010101u;
}

// two of the four 0/1 bytes as 16-bit masks (pair 0: bytes 0 and 1)
template <int PAIR>
__device__ __forceinline__ uint32_t mask2(uint32_t b)
{
    return __byte_perm(b, 0u, PAIR ? 0x4342 : 0x4140) * 0xFFFFu;
}

// One chunk's masks: m = voxel nonzero, x = its value differs from the
// neighbour's (never needed for values 0 and 1, where a change is a zero on one
// side and the count there restarts by itself).
template <bool BIN, int H>
__device__ __forceinline__ void lin_masks(uint32_t v, uint32_t nb, uint32_t (&m)[H], uint32_t (&x)[H])
{
    const uint32_t nz = BIN ? v : nz01(v);
    m[0] = mask2<0>(nz);
    if constexpr (H == 2)
        m[1] = mask2<1>(nz);
    if constexpr (!BIN) {
        const uint32_t df = nz01(v ^ nb);
        x[0] = mask2<0>(df);
        if constexpr (H == 2)
            x[1] = mask2<1>(df);
    }
}

// count of a voxel from the count `c` it has without an event
template <bool BIN>
__device__ __forceinline__ uint32_t lin_count(uint32_t c, uint32_t m, uint32_t x)
{
    return BIN ? c & m : ((c & ~x) | (0x00010001u & x)) & m;
}

// The counts a chunk hands on: forward through dn (in: at its first voxel, out:
// at the voxel after it), backward from "unknown" into en (at the voxel before).
template <bool BIN, int H>
__device__ __forceinline__ void lin_hand_on(const uint32_t (&v)[kLinChunk + 1], uint32_t vp, int len,
                                            uint32_t (&dn)[H], uint32_t (&en)[H])
{
#pragma unroll
    for (int u = 0; u < kLinChunk; u++)
        if (u < len) {
            uint32_t m[H], x[H] = {};
            lin_masks<BIN, H>(v[u], u ? v[u ? u - 1 : 0] : vp, m, x);
#pragma unroll
            for (int h = 0; h < H; h++)
                dn[h] = lin_count<BIN>(dn[h], m[h], x[h]) + 0x00010001u;
        }
#pragma unroll
    for (int u = kLinChunk - 1; u >= 0; u--)
        if (u < len) {
            uint32_t m[H], x[H] = {};
            lin_masks<BIN, H>(v[u], v[u + 1], m, x);
#pragma unroll
            for (int h = 0; h < H; h++)
                en[h] = lin_count<BIN>(en[h], m[h], x[h]) + 0x00010001u;
        }
}

// Both directions of a chunk with the true incoming counts: put(u, counts).
template <bool BIN, int H, class Put>
__device__ __forceinline__ void lin_chunk(const uint32_t (&v)[kLinChunk + 1], uint32_t vp, int len, uint32_t (&dn)[H],
                                          uint32_t (&e)[H], Put &&put)
{
    uint32_t d[kLinChunk][H];
#pragma unroll
    for (int u = 0; u < kLinChunk; u++) {
        uint32_t m[H], x[H] = {};
        lin_masks<BIN, H>(v[u], u ? v[u ? u - 1 : 0] : vp, m, x);
#pragma unroll
        for (int h = 0; h < H; h++) {
            d[u][h] = lin_count<BIN>(dn[h], m[h], x[h]);
            dn[h] = d[u][h] + 0x00010001u;
        }
    }
#pragma unroll
    for (int u = kLinChunk - 1; u >= 0; u--)
        if (u < len) {
            uint32_t m[H], x[H] = {}, r[H];
            lin_masks<BIN, H>(v[u], v[u + 1], m, x);
#pragma unroll
            for (int h = 0; h < H; h++) {
                e[h] = lin_count<BIN>(e[h], m[h], x[h]);
                r[h] = min2(d[u][h], e[h]);
                e[h] += 0x00010001u;
            }
            put(u, r);
        }
}

// Lines along axis 0 of [n][plane], VEC adjacent lines per lane (VEC = 4 where
// plane and the pointers are multiples of 4, else 1), blockDim = (32, segments
// of `seg` positions).  Each thread first runs its segment from "unknown" in
// both directions (what it hands on to the neighbouring segments is the
// smaller of its own count and the incoming one plus its length), then, with
// the true incoming counts, computes both directions chunk by chunk in
// registers and writes each output once.  An event is a zero (count 0) or a
// change between nonzero values (count 1 on both sides).
// Bound by HBM: 1 byte read (twice, the second time from cache) and 2 (4)
// written per voxel; the chunk loops stay rolled, because unrolled they miss
// the instruction cache.
template <int VEC, class OUT>
__global__ void __launch_bounds__(32 * kLinWarps, 2) k_lin(const uint8_t *__restrict__ img, OUT *__restrict__ out,
                                                        long long plane, int n, int seg, pmg_axis_cfg cfg,
                                                        const __grid_constant__ typename TabOf<OUT>::T tab)
{
    constexpr int H = VEC == 4 ? 2 : 1; // 32-bit words of two counts
    constexpr uint32_t kInf2 = (uint32_t)kLinInf * 0x10001u;
    constexpr uint32_t kCap2 = kInf2 + 0x20002000u; // keeps both halves below 2^16 over long lines
    __shared__ uint32_t s_f[kLinWarps][H][32], s_b[kLinWarps][H][32];
    __shared__ uint32_t s_corr[2][H][32];
    extern __shared__ uint32_t s_dyn[]; // backward counts of the chunks [nw][kLinChunks][H][32], then the table
    const int lane = threadIdx.x, w = threadIdx.y, nw = blockDim.y;
    uint32_t *s_en = s_dyn + w * kLinChunks * H * 32 + lane;
    float *s_tab = reinterpret_cast<float *>(s_dyn + nw * kLinChunks * H * 32);
    if constexpr (sizeof(OUT) == 4)
        for (int q = w * 32 + lane; q <= n; q += nw * 32)
            s_tab[q] = tab.v[q];
    const long long line = ((long long)blockIdx.x * 32 + lane) * VEC;
    const bool live = line < plane;
    const uint8_t *in = img + (live ? line : 0);
    auto row = [&](int i) -> uint32_t {
        if constexpr (VEC == 4)
            return __ldg(reinterpret_cast<const uint32_t *>(in + i * plane));
        else
            return __ldg(in + i * plane);
    };
    const int i0 = w * seg, i1 = min(n, i0 + seg);
    const int nc = (i1 - i0 + kLinChunk - 1) / kLinChunk;
    // periodic correctors: the count at the last voxel from the first zero of
    // the wrapped line, and at the first voxel from the last one
    if (cfg.periodic && (w == 0 || w == nw - 1)) {
        for (int side = 0; side < 2; side++) {
            if (side == 0 ? w != 0 : w != nw - 1)
                continue;
            int pos[VEC];
            const int lo = side == 0 ? cfg.f_lo : cfg.l_lo, hi = side == 0 ? n : n - cfg.l_hi;
#pragma unroll
            for (int q = 0; q < VEC; q++)
                pos[q] = -1;
            for (int t = 0; t < hi - lo; t += 4) {
                uint32_t r[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    r[u] = t + u < hi - lo ? row(side == 0 ? lo + t + u : hi - 1 - t - u) : 0xffffffffu;
                bool open = false;
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int q = 0; q < VEC; q++)
                        if (pos[q] < 0 && ((r[u] >> (8 * q)) & 0xffu) == 0)
                            pos[q] = t + u;
#pragma unroll
                for (int q = 0; q < VEC; q++)
                    open |= pos[q] < 0;
                if (!__any_sync(0xffffffffu, open && live))
                    break;
            }
            uint32_t c[VEC];
#pragma unroll
            for (int q = 0; q < VEC; q++) {
                if (pos[q] < 0)
                    c[q] = kLinInf;
                else if (side == 0) // first zero F: the upper corrector F + a_u
                    c[q] = (uint32_t)(lo + pos[q] + cfg.a_u);
                else // last zero L: the lower corrector n - L + a_l
                    c[q] = (uint32_t)(n - (hi - 1 - pos[q]) + cfg.a_l);
            }
#pragma unroll
            for (int h = 0; h < H; h++)
                s_corr[side][h][lane] = VEC == 4 ? c[2 * h % VEC] | (c[(2 * h + 1) % VEC] << 16) : c[0];
        }
    }
    uint32_t v[kLinChunk + 1];
    // a chunk's words and the next one (the last voxel again past the line's
    // end); true when they all are 0 or 1
    auto load = [&](int a, uint32_t vp) -> bool {
        uint32_t big = vp;
#pragma unroll
        for (int u = 0; u <= kLinChunk; u++) {
            v[u] = row(min(a + u, n - 1));
            big |= v[u];
        }
        return !__any_sync(0xffffffffu, (big & 0xfefefefeu) != 0);
    };
    // counts handed on, from unknown incoming ones
    uint32_t dn[H], en[H];
#pragma unroll
    for (int h = 0; h < H; h++)
        dn[h] = kInf2;
    uint32_t vp = row(i0 > 0 ? i0 - 1 : 0);
#pragma unroll 1
    for (int c = 0; c < nc; c++) {
        const int a = i0 + c * kLinChunk, len = min(kLinChunk, i1 - a);
        const bool bin = load(a, vp);
#pragma unroll
        for (int h = 0; h < H; h++)
            en[h] = kInf2;
        if (bin)
            lin_hand_on<true, H>(v, vp, len, dn, en);
        else
            lin_hand_on<false, H>(v, vp, len, dn, en);
#pragma unroll
        for (int h = 0; h < H; h++)
            s_en[(c * H + h) * 32] = en[h];
        vp = v[kLinChunk - 1]; // (a short chunk is the line's last)
    }
    // the segment's backward count: chunk by chunk from its high end
#pragma unroll
    for (int h = 0; h < H; h++)
        en[h] = kInf2;
    for (int c = nc - 1; c >= 0; c--) {
        const uint32_t len = (uint32_t)min(kLinChunk, i1 - i0 - c * kLinChunk) * 0x10001u;
#pragma unroll
        for (int h = 0; h < H; h++)
            en[h] = min2(s_en[(c * H + h) * 32], en[h] + len);
    }
#pragma unroll
    for (int h = 0; h < H; h++) {
        s_f[w][h][lane] = dn[h];
        s_b[w][h][lane] = min2(en[h], kCap2);
    }
    __syncthreads();
    // the true incoming counts of this segment
#pragma unroll
    for (int h = 0; h < H; h++) {
        dn[h] = cfg.periodic ? s_corr[1][h][lane] : kInf2;
        en[h] = cfg.periodic ? s_corr[0][h][lane] : kInf2;
        for (int q = 0; q < w; q++)
            dn[h] = min2(min2(s_f[q][h][lane], dn[h] + (uint32_t)seg * 0x10001u), kCap2);
        for (int q = nw - 1; q > w; q--) {
            const uint32_t len = (uint32_t)(min(n, (q + 1) * seg) - q * seg) * 0x10001u;
            en[h] = min2(min2(s_b[q][h][lane], en[h] + len), kCap2);
        }
    }
    // the backward count above every chunk
    for (int c = nc - 1; c >= 0; c--) {
        const uint32_t len = (uint32_t)min(kLinChunk, i1 - i0 - c * kLinChunk) * 0x10001u;
#pragma unroll
        for (int h = 0; h < H; h++) {
            const uint32_t own = s_en[(c * H + h) * 32];
            s_en[(c * H + h) * 32] = en[h];
            en[h] = min2(own, en[h] + len);
        }
    }
    vp = row(i0 > 0 ? i0 - 1 : 0);
#pragma unroll 1
    for (int c = 0; c < nc; c++) {
        const int a = i0 + c * kLinChunk, len = min(kLinChunk, i1 - a);
        const bool bin = load(a, vp);
#pragma unroll
        for (int h = 0; h < H; h++)
            en[h] = s_en[(c * H + h) * 32];
        OUT *o = out + (long long)a * plane + line;
        auto put = [&](int u, const uint32_t (&r)[H]) {
            if (!live)
                return;
            OUT *q = o + u * plane;
            if constexpr (sizeof(OUT) == 2) {
                if constexpr (VEC == 4)
                    *reinterpret_cast<uint2 *>(q) = make_uint2(r[0], r[H - 1]);
                else
                    *q = (OUT)r[0];
            } else {
                auto val = [&](uint32_t k) { return k <= (uint32_t)n ? s_tab[k] : FLT_MAX; };
                if constexpr (VEC == 4)
                    *reinterpret_cast<float4 *>(q) = make_float4(val(r[0] & 0xffffu), val(r[0] >> 16),
                                                                 val(r[H - 1] & 0xffffu), val(r[H - 1] >> 16));
                else
                    *q = (OUT)val(r[0] & 0xffffu);
            }
        };
        if (bin)
            lin_chunk<true, H>(v, vp, len, dn, en, put);
        else
            lin_chunk<false, H>(v, vp, len, dn, en, put);
        vp = v[kLinChunk - 1];
    }
}

// The linear pass as counts needs correctors that are counts themselves.
bool lin_ok(int n, const pmg_axis_cfg &c)
{
    if (n > kLinMaxLine)
        return false;
    if (!c.periodic)
        return true;
    // every index in range, and both correctors of every line in [0, kLinInf)
    return c.f_lo >= 0 && c.l_lo >= 0 && c.l_hi >= 0 && c.l_lo + c.l_hi <= n && (long long)c.f_lo + c.a_u >= 0 &&
           (long long)c.l_hi + 1 + c.a_l >= 0 && 2LL * n + std::max(c.a_u, c.a_l) < kLinInf;
}

template <class OUT>
static int launch_lin_t(const uint8_t *img, OUT *out, const int64_t *shape, float res, const pmg_axis_cfg &cfg,
                        cudaStream_t st)
{
    const int n = (int)shape[0];
    const long long plane = (long long)shape[1] * shape[2];
    // segments of whole chunks: 8 per line, 16 on lines beyond 1024
    const int parts = n > 8 * kLinChunk * kLinChunks ? kLinWarps : 8;
    const int seg = ((n + parts - 1) / parts + kLinChunk - 1) / kLinChunk * kLinChunk;
    const dim3 block(32, (unsigned)((n + seg - 1) / seg));
    typename TabOf<OUT>::T tab;
    size_t smem = sizeof(uint32_t) * (size_t)block.y * kLinChunks * 2 * 32;
    if constexpr (sizeof(OUT) == 4) {
        // the reference's running sum of res, squared (_distance.hpp:135-182)
        float d = 0.0f;
        for (int k = 0; k <= n; k++) {
            volatile float q = d * d;
            tab.v[k] = q == INFINITY ? FLT_MAX : (float)q;
            volatile float nd = d + res;
            d = nd;
        }
        smem += sizeof(float) * (size_t)(n + 1);
    }
    const bool quads = !(plane & 3) && !(reinterpret_cast<uintptr_t>(img) & 3) &&
                       !(reinterpret_cast<uintptr_t>(out) & (4 * sizeof(OUT) - 1));
    if (smem > 36 * 1024) { // (with the static arrays above the default limit)
        PMG_CUDA(cudaFuncSetAttribute(k_lin<4, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        PMG_CUDA(cudaFuncSetAttribute(k_lin<1, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    }
    const int ps__ = prof_begin("k_lin", st);
    if (quads)
        k_lin<4, OUT><<<(unsigned)((plane / 4 + 31) / 32), block, smem, st>>>(img, out, plane, n, seg, cfg, tab);
    else
        k_lin<1, OUT><<<(unsigned)((plane + 31) / 32), block, smem, st>>>(img, out, plane, n, seg, cfg, tab);
    prof_end(ps__, (double)plane * n * (1 + sizeof(OUT)), st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

int launch_lin_counts(const uint8_t *img, uint16_t *out, const int64_t *shape, const pmg_axis_cfg &cfg,
                      cudaStream_t st)
{
    return launch_lin_t<uint16_t>(img, out, shape, 1.0f, cfg, st);
}

int launch_lin_float(const uint8_t *img, float *out, const int64_t *shape, float res, const pmg_axis_cfg &cfg,
                     cudaStream_t st)
{
    return launch_lin_t<float>(img, out, shape, res, cfg, st);
}

// ---------------------------------------------------------------------------
// envelope passes
// ---------------------------------------------------------------------------
// Heights of kBig and more count as absent; kBig + 2 * kMaxStep stays below
// 2^16, and (kMaxStep + 1)^2 is above every height below kBig.
constexpr uint32_t kBig = 60000u, kMaxStep = 245u;
constexpr uint32_t kBig2 = kBig * 0x10001u;

// Wide pores: all steps take up to 17 ps a voxel (512^3: 2.3 ms a pass), and lines
// with a voxel left out of range go to the float envelope (15 to 50 ps) all the
// same.  So where most threads of a block (warp) still hold positions without any
// height in range after 32 steps, or a quarter of them after 64, its lines are left
// to the envelope at once (only where heights may exceed the range at all and the
// line reaches beyond it).  512^3, both passes, ms, all steps and whole lines
// afterwards, envelope alone, now: no solid 13.2, 3.8, 2.1; ball of radius 51 in the
// middle 18.0, 9.8, 8.5; points 160 voxels apart 13.2, 6.0, 6.1, 40 apart 23.6, 14.1,
// 14.0, 10 apart 2.6, 7.3, 2.6; cavity of radius 230 1.4, 4.8, 1.4.
__device__ __forceinline__ uint32_t first_stop(uint32_t last) { return min(last, 31u); }
__device__ __forceinline__ uint32_t next_stop(uint32_t stop, uint32_t last) { return stop < 32 ? min(last, 63u) : last; }
__device__ __forceinline__ bool give_up(uint32_t stop, int lost, int threads)
{
    return stop < 32 ? 4 * lost > 3 * threads : 4 * lost > threads;
}

// (count, count) -> (K, K), absent counts -> kBig; the counted voxels are 2^shift
// of the pass's own (shift <= kMaxShift)
constexpr int kMaxShift = 16;

__device__ __forceinline__ uint32_t square2(uint32_t c, int shift)
{
    const uint32_t a = min(min(c & 0xffffu, 255u) << shift, kMaxStep), b = min(min(c >> 16, 255u) << shift, kMaxStep);
    return min(a * a, kBig) | (min(b * b, kBig) << 16);
}

// heights -> (K, K)
__device__ __forceinline__ uint32_t pack_heights(float f0, float f1, float inv_a)
{
    return pack_float2(fminf(fmul(f0, inv_a), (float)kBig), fminf(fmul(f1, inv_a), (float)kBig));
}

// height of an integer minimum
__device__ __forceinline__ float par_value(float k, float a) { return k >= (float)kBig ? FLT_MAX : fmul(k, a); }

// larger of the two halves
__device__ __forceinline__ uint32_t hmax(uint32_t v) { return max(v & 0xffffu, v >> 16); }

// smallest value of P positions
template <int P>
__device__ __forceinline__ uint32_t hmin(const uint32_t (&g)[P])
{
    uint32_t m = g[0];
#pragma unroll
    for (int p = 1; p < P; p++)
        m = min2(m, g[p]);
    return min(m & 0xffffu, m >> 16);
}

// Steps k and k + 1 on P positions in registers, given the two values on
// either side before step k; returns the maxima of the first `valid` results.
template <int P>
__device__ __forceinline__ uint32_t par_steps(uint32_t (&g)[P], uint32_t l2, uint32_t l1, uint32_t r1, uint32_t r2,
                                              uint32_t k, int valid)
{
    const uint32_t c = (2 * k - 1) * 0x10001u, d = c + 0x00020002u;
    // the neighbours' end values after step k
    uint32_t prev = l1, left = __viaddmin_u16x2(min2(l2, g[0]), c, l1);
    uint32_t right = __viaddmin_u16x2(min2(g[P - 1], r2), c, r1);
#pragma unroll
    for (int p = 0; p < P; p++) {
        const uint32_t cur = g[p];
        g[p] = __viaddmin_u16x2(prev, c, __viaddmin_u16x2(p + 1 < P ? g[p + 1 < P ? p + 1 : p] : r1, c, cur));
        prev = cur;
    }
    prev = left;
#pragma unroll
    for (int p = 0; p < P; p++) {
        const uint32_t cur = g[p];
        g[p] = __viaddmin_u16x2(prev, d, __viaddmin_u16x2(p + 1 < P ? g[p + 1 < P ? p + 1 : p] : right, d, cur));
        prev = cur;
    }
    uint32_t mx = 0;
    if (valid >= P) {
#pragma unroll
        for (int p = 0; p < P; p += 2)
            mx = __vimax3_u16x2(mx, g[p], g[p + 1]);
    } else {
#pragma unroll
        for (int p = 0; p < P; p++)
            if (p < valid)
                mx = max2(mx, g[p]);
    }
    return mx;
}

// How far the imports beyond a periodic line's ends can reach into it, and
// lines that need the float envelope: byte 0 (1) is one more than the last
// position from the low (high) end whose minimum exceeds the squared distance
// to the first import, byte 0 = kWholeLine the whole line.  g: the minima of
// positions x0 ... of two lines, mx: their maxima (of valid positions); bytes
// 0-1 for the line in the low halves, 2-3 for the other.
template <int P>
__device__ __forceinline__ uint32_t line_reach(const uint32_t (&g)[P], uint32_t mx, int x0, int n, int periodic,
                                               int wide, bool second)
{
    const uint32_t big = hmax(mx);
    const int last = min(x0 + P, n) - 1;
    uint32_t lo0 = 0, lo1 = 0, hi0 = 0, hi1 = 0;
    if (periodic && big > (uint32_t)((x0 + 1) * (x0 + 1)))
#pragma unroll
        for (int p = 0; p < P; p++) {
            const uint32_t e = (uint32_t)(x0 + p + 1);
            if (x0 + p < n && e <= kMaxStep) {
                if ((g[p] & 0xffffu) > e * e)
                    lo0 = e;
                if ((g[p] >> 16) > e * e)
                    lo1 = e;
            }
        }
    if (periodic && big > (uint32_t)((n - last) * (n - last)))
#pragma unroll
        for (int p = P - 1; p >= 0; p--) {
            const uint32_t e = (uint32_t)(n - x0 - p);
            if (x0 + p < n && e <= kMaxStep) {
                if ((g[p] & 0xffffu) > e * e)
                    hi0 = e;
                if ((g[p] >> 16) > e * e)
                    hi1 = e;
            }
        }
    if (big >= kBig && wide) {
        if ((mx & 0xffffu) >= kBig)
            lo0 = kWholeLine;
        if ((mx >> 16) >= kBig)
            lo1 = kWholeLine;
    }
    return lo0 | (hi0 << 8) | (second ? (lo1 << 16) | (hi1 << 24) : 0u);
}

// Strided pass along axis 1 of [n0][n][s2] in at most `last` steps: one thread block per plane and
// LN * VEC adjacent lines (VEC = 2: two lines per thread, s2 even), thread
// group q of LN on positions [q P, (q + 1) P) of its lines, heights in
// registers.  Groups hand their end values on through shared memory, one
// barrier per step.  Lines beyond 512 voxels take LN = 16, so that two blocks
// share an SM and one loads while the other computes.
// Bound by the packed add-min pipe (two instructions per pair of voxels and
// distance).
template <class T, int P, int VEC, int LN>
__global__ void __launch_bounds__(P == 32 ? 512 : 32 * P, P == 32 ? 2 : 1)
    k_par_cols(const T *__restrict__ D, float *__restrict__ out, int n, int s2, float a, float inv_a, int shift, int last,
               int periodic, int wide, uint16_t *__restrict__ flag)
{
    extern __shared__ uint32_t s_end[]; // [2][groups][4][LN]
    const int l = threadIdx.x % LN, w = threadIdx.x / LN, nw = blockDim.x / LN;
    const int k0 = (blockIdx.x * LN + l) * VEC;
    const int x0 = w * P;
    const bool live = k0 < s2 && x0 < n;
    const long long base = (long long)blockIdx.y * n * s2 + k0;
    uint32_t g[P];
    const T *src = D + base + (long long)x0 * s2;
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int p = 0; p < P; p++) {
            uint32_t c = 0xffffffffu;
            if (live && x0 + p < n) {
                if constexpr (VEC == 2)
                    c = __ldg(reinterpret_cast<const uint32_t *>(src + (long long)p * s2));
                else
                    c = (uint32_t)__ldg(src + (long long)p * s2) | 0xffff0000u;
            }
            g[p] = c;
        }
#pragma unroll
        for (int p = 0; p < P; p++)
            g[p] = square2(g[p], shift);
    } else {
        float f[P][VEC];
#pragma unroll
        for (int p = 0; p < P; p++)
#pragma unroll
            for (int v = 0; v < VEC; v++)
                f[p][v] = live && x0 + p < n ? __ldg(src + (long long)p * s2 + v) : FLT_MAX;
#pragma unroll
        for (int p = 0; p < P; p++)
            g[p] = pack_heights(f[p][0], VEC == 2 ? f[p][VEC - 1] : FLT_MAX, inv_a);
    }
    uint32_t mx = 0;
#pragma unroll
    for (int p = 0; p < P; p++)
        if (x0 + p < n)
            mx = max2(mx, g[p]);
    if (!live)
        mx = 0;
    if (VEC == 1)
        mx &= 0xffffu;
    // two steps per round: the neighbours' two end values on either side
    for (uint32_t k = 1; k <= (uint32_t)last; k += 2) {
        uint32_t *e = s_end + (size_t)((k >> 1) & 1) * nw * 4 * LN + l;
        e[(w * 4 + 0) * LN] = g[0];
        e[(w * 4 + 1) * LN] = g[1];
        e[(w * 4 + 2) * LN] = g[P - 2];
        e[(w * 4 + 3) * LN] = g[P - 1];
        const bool open = hmax(mx) > k * k;
        if (!__syncthreads_or(open))
            break;
        if (wide && n > (int)kMaxStep && (k == 33 || k == 65)) {
            const int lost = __syncthreads_count(hmax(mx) >= kBig);
            if (give_up(k - 2, lost, (n + P - 1) / P * LN)) {
                if (w == 0 && live) {
                    uint16_t *fl = flag + (long long)blockIdx.y * s2 + k0;
                    if constexpr (VEC == 2)
                        *reinterpret_cast<uint32_t *>(fl) = kWholeLine * 0x10001u;
                    else
                        *fl = kWholeLine;
                }
                return;
            }
        }
        if (!__any_sync(0xffffffffu, open))
            continue; // this warp's values are final
        uint32_t l2 = kBig2, l1 = kBig2, r1 = kBig2, r2 = kBig2;
        if (w > 0) {
            l2 = e[(w * 4 - 2) * LN];
            l1 = e[(w * 4 - 1) * LN];
        }
        if (w + 1 < nw) {
            r1 = e[(w * 4 + 4) * LN];
            r2 = e[(w * 4 + 5) * LN];
        }
        mx = par_steps<P>(g, l2, l1, r1, r2, k, n - x0);
        if (!live)
            mx = 0;
        if (VEC == 1)
            mx &= 0xffffu;
    }
    if (live) {
        float *dst = out + base + (long long)x0 * s2;
#pragma unroll
        for (int p = 0; p < P; p++) {
            if (x0 + p >= n)
                break;
            const float f0 = par_value(lo_float(g[p]), a);
            if constexpr (VEC == 2) {
                const float f1 = par_value(hi_float(g[p]), a);
                *reinterpret_cast<float2 *>(dst + (long long)p * s2) = make_float2(f0, f1);
            } else {
                dst[(long long)p * s2] = f0;
            }
        }
    }
    if (!flag)
        return;
    __syncthreads();
    s_end[w * LN + l] = live ? line_reach<P>(g, mx, x0, n, periodic, wide, VEC == 2) : 0u;
    __syncthreads();
    if (w == 0 && live) {
        uint32_t need = 0;
        for (int q = 0; q < nw; q++)
            need = __vmaxu4(need, s_end[q * LN + l]);
        uint16_t *fl = flag + (long long)blockIdx.y * s2 + k0;
        if constexpr (VEC == 2)
            *reinterpret_cast<uint32_t *>(fl) = need;
        else
            *fl = (uint16_t)need;
    }
}

// Contiguous pass: one warp per pair of rows, lane l on positions [l P, (l +
// 1) P), neighbouring values by shuffles; the rows pass through shared memory
// (one word per position pair, padded by one word per P) so that global
// loads and stores stay coalesced.
constexpr int kRowWarps = 8;

template <int P>
__global__ void __launch_bounds__(32 * kRowWarps, 4) k_par_rows(const float *__restrict__ fin, float *__restrict__ fout,
                                                             long long nrows, int n, float a, float inv_a,
                                                             int periodic, int wide, int form,
                                                             uint16_t *__restrict__ flag)
{
    constexpr int kWords = 32 * P + 32;
    extern __shared__ uint32_t s_rows[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t *row = s_rows + w * kWords;
    const long long pairs = (nrows + 1) >> 1;
    const bool vec4 = !(n & 3) && !((reinterpret_cast<uintptr_t>(fin) | reinterpret_cast<uintptr_t>(fout)) & 15);
    const uint32_t last = min(kMaxStep, (uint32_t)n - 1);
    auto pack = [&](float f0, float f1) -> uint32_t { return pack_heights(f0, f1, inv_a); };
    auto slot = [](int c) { return c + c / P; };
    for (long long r = blockIdx.x * (long long)kRowWarps + w; r < pairs; r += (long long)gridDim.x * kRowWarps) {
        const bool two = 2 * r + 1 < nrows;
        const float *in0 = fin + 2 * r * n, *in1 = in0 + (two ? n : 0);
        if (vec4) {
#pragma unroll 2
            for (int t = 0; t < (P + 3) / 4; t++) {
                const int c = (t * 32 + lane) * 4;
                if (c < n) {
                    const float4 f0 = __ldg(reinterpret_cast<const float4 *>(in0 + c));
                    const float4 f1 = __ldg(reinterpret_cast<const float4 *>(in1 + c));
                    row[slot(c)] = pack(f0.x, f1.x);
                    row[slot(c + 1)] = pack(f0.y, f1.y);
                    row[slot(c + 2)] = pack(f0.z, f1.z);
                    row[slot(c + 3)] = pack(f0.w, f1.w);
                }
            }
        } else {
#pragma unroll 4
            for (int t = 0; t < P; t++) {
                const int c = t * 32 + lane;
                if (c < n)
                    row[slot(c)] = pack(in0[c], in1[c]);
            }
        }
        __syncwarp();
        const int x0 = lane * P;
        uint32_t g[P], mx = 0;
#pragma unroll
        for (int p = 0; p < P; p++) {
            g[p] = x0 + p < n ? row[lane * (P + 1) + p] : kBig2;
            if (x0 + p < n)
                mx = max2(mx, g[p]);
        }
        bool left = false; // to the envelope
        uint32_t k = 1;
        for (uint32_t stop = first_stop(last);; stop = next_stop(stop, last)) {
            bool done = false;
            for (; k <= stop; k += 2) {
                done = !__any_sync(0xffffffffu, hmax(mx) > k * k);
                if (done)
                    break;
                uint32_t l1 = __shfl_up_sync(0xffffffffu, g[P - 1], 1), l2 = __shfl_up_sync(0xffffffffu, g[P - 2], 1);
                uint32_t r1 = __shfl_down_sync(0xffffffffu, g[0], 1), r2 = __shfl_down_sync(0xffffffffu, g[1], 1);
                if (lane == 0)
                    l1 = l2 = kBig2;
                if (lane == 31)
                    r1 = r2 = kBig2;
                mx = par_steps<P>(g, l2, l1, r1, r2, k, n - x0);
            }
            if (done || k > last)
                break;
            left = wide && n > (int)kMaxStep &&
                   give_up(stop, __popc(__ballot_sync(0xffffffffu, hmax(mx) >= kBig)), (n + P - 1) / P);
            if (left || !__any_sync(0xffffffffu, hmin<P>(g) < kBig))
                break;
        }
        if (left) {
            if (lane < (two ? 2 : 1))
                flag[2 * r + lane] = kWholeLine;
            __syncwarp();
            continue;
        }
#pragma unroll
        for (int p = 0; p < P; p++)
            if (x0 + p < n)
                row[lane * (P + 1) + p] = g[p];
        __syncwarp();
        auto value = [&](float k) -> float {
            const float f = par_value(k, a);
            return form == PMG_EDT_DIST ? __fsqrt_rn(f) : f;
        };
        float *o0 = fout + 2 * r * n, *o1 = o0 + n;
        if (vec4) {
#pragma unroll 2
            for (int t = 0; t < (P + 3) / 4; t++) {
                const int c = (t * 32 + lane) * 4;
                if (c < n) {
                    const uint32_t q0 = row[slot(c)], q1 = row[slot(c + 1)], q2 = row[slot(c + 2)],
                                   q3 = row[slot(c + 3)];
                    *reinterpret_cast<float4 *>(o0 + c) = make_float4(value(lo_float(q0)), value(lo_float(q1)),
                                                                      value(lo_float(q2)), value(lo_float(q3)));
                    if (two)
                        *reinterpret_cast<float4 *>(o1 + c) =
                            make_float4(value(hi_float(q0)), value(hi_float(q1)), value(hi_float(q2)), value(hi_float(q3)));
                }
            }
        } else {
#pragma unroll 4
            for (int t = 0; t < P; t++) {
                const int c = t * 32 + lane;
                if (c < n) {
                    const uint32_t q = row[slot(c)];
                    o0[c] = value(lo_float(q));
                    if (two)
                        o1[c] = value(hi_float(q));
                }
            }
        }
        if (flag) {
            uint32_t need = x0 < n ? line_reach<P>(g, mx, x0, n, periodic, wide, two) : 0u;
            if (__any_sync(0xffffffffu, need != 0)) {
                uint32_t all = 0;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    all |= __reduce_max_sync(0xffffffffu, (need >> (8 * q)) & 0xffu) << (8 * q);
                need = all;
            }
            if (lane == 0) {
                flag[2 * r] = (uint16_t)need;
                if (two)
                    flag[2 * r + 1] = (uint16_t)(need >> 16);
            }
        }
        __syncwarp();
    }
}

// log2 of the ratio of two power-of-two voxel sizes, -1 when a < b or it is too large
static int size_shift(float a, float b)
{
    int ea = 0, eb = 0;
    frexpf(a, &ea);
    frexpf(b, &eb);
    return ea < eb || ea - eb > kMaxShift ? -1 : ea - eb;
}

// Which passes run on the lattice, and from what (edt_internal.cuh).
LatticePlan lattice_plan(const int64_t *shape, const float *res, const pmg_axis_cfg *cfg)
{
    LatticePlan P{};
    const int n1 = (int)shape[1], n2 = (int)shape[2];
    // (window_path_ok of one voxel: a power of two)
    if (!window_path_ok(res[0], 1) || !window_path_ok(res[1], 1) || !window_path_ok(res[2], 1))
        return P;
    P.shift = size_shift(res[0], res[1]);
    P.cols = n1 <= kScanMaxLine && P.shift >= 0;
    P.counts = P.cols && lin_ok((int)shape[0], cfg[0]);
    P.rows = n2 <= kScanMaxLine && size_shift(res[0], res[2]) >= 0 && size_shift(res[1], res[2]) >= 0;
    // whether a finite value of a pass can reach kBig (counts reach n0, or the
    // correctors of a wrapped line, which are distances to one of its zeros)
    const double m0 = ((double)shape[0] + (cfg[0].periodic ? std::max(0, std::max(cfg[0].a_u, cfg[0].a_l)) : 0)) * res[0];
    const double m1 = m0 * m0 + (double)n1 * n1 * res[1] * res[1], m2 = m1 + (double)n2 * n2 * res[2] * res[2];
    P.wide1 = m1 >= (double)kBig * res[1] * res[1];
    P.wide2 = m2 >= (double)kBig * res[2] * res[2];
    return P;
}

template <class T, int P, int LN>
static void cols_p(const T *D, float *out, int n0, int n, int s2, float a, int shift, int last, int periodic, int wide,
                   uint16_t *flag, cudaStream_t st)
{
    // whole warps (the last group may lie past the line's end)
    const int groups = ((n + P - 1) / P + 32 / LN - 1) / (32 / LN) * (32 / LN);
    const size_t smem = (size_t)groups * 8 * LN * sizeof(uint32_t);
    const unsigned threads = (unsigned)(groups * LN);
    if (!(s2 & 1))
        k_par_cols<T, P, 2, LN><<<dim3((unsigned)((s2 / 2 + LN - 1) / LN), (unsigned)n0), threads, smem, st>>>(
            D, out, n, s2, a, 1.0f / a, shift, last, periodic, wide, flag);
    else
        k_par_cols<T, P, 1, LN><<<dim3((unsigned)((s2 + LN - 1) / LN), (unsigned)n0), threads, smem, st>>>(
            D, out, n, s2, a, 1.0f / a, shift, last, periodic, wide, flag);
}

template <class T>
static int cols_run(const T *D, float *out, int n0, int n, int s2, float a, int shift, int last, int periodic, int wide,
                    uint16_t *flag, cudaStream_t st)
{
    const int ps__ = prof_begin("k_par_cols", st);
    if (n <= 64)
        cols_p<T, 8, 32>(D, out, n0, n, s2, a, shift, last, periodic, wide, flag, st);
    else if (n <= 256)
        cols_p<T, 16, 32>(D, out, n0, n, s2, a, shift, last, periodic, wide, flag, st);
    else if (n <= 512)
        cols_p<T, 32, 32>(D, out, n0, n, s2, a, shift, last, periodic, wide, flag, st);
    else
        cols_p<T, 32, 16>(D, out, n0, n, s2, a, shift, last, periodic, wide, flag, st);
    prof_end(ps__, (double)n0 * n * s2 * (sizeof(T) + 4), st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

template <int P>
static void rows_p(const float *fin, float *fout, long long nrows, int n, float a, int periodic, int wide, int form,
                   uint16_t *flag, cudaStream_t st)
{
    const size_t smem = sizeof(uint32_t) * (size_t)kRowWarps * (32 * P + 32);
    const long long pairs = (nrows + 1) >> 1;
    k_par_rows<P><<<grid_for(pairs, kRowWarps, 152LL * 64), 32 * kRowWarps, smem, st>>>(fin, fout, nrows, n, a, 1.0f / a,
                                                                                    periodic, wide, form, flag);
}

// Pass along axis 1 of planes [lo, lo + planes) of a volume X of power-of-two voxels,
// from heights; only values up to T (times the squared size) matter, larger ones
// come out as anything above.
bool cols_capped_ok(const int64_t *X, float res, int T)
{
    return tune_value(kTuneEdtPath) == 0 && window_path_ok(res, (int)X[1]) && T >= 0 && T < (int)kBig;
}

int launch_cols_capped(const float *fin, float *fout, const int64_t *X, int lo, int planes, float res, int T,
                       cudaStream_t st)
{
    int W = 0;
    while ((W + 1) * (W + 1) <= T)
        W++;
    const long long at = (long long)lo * X[1] * X[2];
    return cols_run(fin + at, fout + at, planes, (int)X[1], (int)X[2], res * res, 0, std::min(W + 1, (int)X[1] - 1), 0, 0,
                    nullptr, st);
}

// What a lattice pass left over: the ends of periodic lines, and whole lines.
template <class T>
static int rest(const T *in, float *out, const Lines &Ls, float res, float resh, const pmg_axis_cfg &cfg, int num_hull,
                int form, uint16_t *flag, int whole, cudaStream_t st)
{
    if (cfg.periodic)
        PMG_TRY(launch_lattice_ends(in, out, Ls, res, resh, cfg, num_hull, form, flag, whole, st));
    return whole ? launch_whole(in, out, Ls, res, resh, cfg, num_hull, form, MorphEpi{}, flag, nullptr, st) : PMG_OK;
}

// (a hull segment of one voxel without a solid gives the reference's phantom
// import: its lines are whole ones)
static bool phantom(const pmg_axis_cfg &c, int n) { return c.periodic && (n - c.hf_lo < 2 || n - c.hb_hi < 2); }

// Pass along axis 1 from counts or heights to `out`.
int lattice_cols(const LatticePlan &P, const void *in, float *out, const int64_t *shape, const float *res,
                 const pmg_axis_cfg *cfg, int num_hull, uint16_t *flags, cudaStream_t st)
{
    const int n0 = (int)shape[0], n1 = (int)shape[1], n2 = (int)shape[2];
    const float a = res[1] * res[1];
    const int per = cfg[1].periodic ? 1 : 0, last = std::min((int)kMaxStep, n1 - 1);
    const int whole = P.wide1 || phantom(cfg[1], n1);
    uint16_t *fl = per || whole ? flags : nullptr;
    const Lines Ls = all_lines(shape, 1);
    if (P.counts) {
        const uint16_t *D = (const uint16_t *)in;
        PMG_TRY(cols_run(D, out, n0, n1, n2, a, P.shift, last, per, whole, fl, st));
        return rest(D, out, Ls, res[1], res[0], cfg[1], num_hull, PMG_EDT_SQUARED, fl, whole, st);
    }
    const float *D = (const float *)in;
    PMG_TRY(cols_run(D, out, n0, n1, n2, a, 0, last, per, whole, fl, st));
    return rest(D, out, Ls, res[1], res[1], cfg[1], num_hull, PMG_EDT_SQUARED, fl, whole, st);
}

// Pass along axis 2.
int lattice_rows(const LatticePlan &P, const float *in, float *out, const int64_t *shape, const float *res,
                 const pmg_axis_cfg *cfg, int num_hull, int form, uint16_t *flags, cudaStream_t st)
{
    const int n2 = (int)shape[2];
    const float a = res[2] * res[2];
    const int per = cfg[2].periodic ? 1 : 0, whole = P.wide2 || phantom(cfg[2], n2);
    uint16_t *fl = per || whole ? flags : nullptr;
    const long long nrows = (long long)shape[0] * shape[1];
    const int ps__ = prof_begin("k_par_rows", st);
    if (n2 <= 64)
        rows_p<2>(in, out, nrows, n2, a, per, whole, form, fl, st);
    else if (n2 <= 128)
        rows_p<4>(in, out, nrows, n2, a, per, whole, form, fl, st);
    else if (n2 <= 256)
        rows_p<8>(in, out, nrows, n2, a, per, whole, form, fl, st);
    else if (n2 <= 512)
        rows_p<16>(in, out, nrows, n2, a, per, whole, form, fl, st);
    else
        rows_p<32>(in, out, nrows, n2, a, per, whole, form, fl, st);
    prof_end(ps__, (double)nrows * n2 * 8, st);
    PMG_CHECK_LAUNCH();
    return rest(in, out, all_lines(shape, 2), res[2], res[2], cfg[2], num_hull, form, fl, whole, st);
}

} // namespace pmg
