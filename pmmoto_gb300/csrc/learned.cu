// Learned radius schedule: the small 3-D CNN that predicts a drainage
// curve from a downsampled distance field.  No counterpart in the
// reference (its drainage loop, equilibrium_distribution.py:93-128, sweeps
// every radius); the network only proposes which radii the exact loop
// evaluates.
//
// Convolutions (3x3x3, stride 2, padding 1, channels-last bf16 activations)
// are implicit GEMMs on the 5th-generation tensor cores:
//
//   forward   D[pos_out, c_out] = sum_{tap, c_in} X[pos_in(pos_out, tap), c_in] W[c_out, tap, c_in]
//   dgrad     D[pos_in, c_in]   = sum_{tap, c_out} dZ[pos_out(pos_in, tap), c_out] W[c_out, tap, c_in]
//   wgrad     D[(tap, c_in), c_out] = sum_{pos_out} X[pos_in(pos_out, tap), c_in] dZ[pos_out, c_out]
//
// One CTA of 128 threads computes 128 x N tiles (N = 16, 32 or 64 output
// columns) with the fp32 accumulator in tensor memory.  The K loop runs in
// chunks of 64 bf16: all threads gather the chunk's operands with 16-byte
// cp.async (the im2col gather, zero-filled outside the volume) into one of
// three shared-memory stages, two chunks ahead of the one elected thread that
// issues four tcgen05.mma (K = 16 each) and commits them to the stage's
// mbarrier.  The epilogue reads the accumulator with tcgen05.ld (thread t owns
// row t) and applies bias + ReLU (forward), the ReLU mask of the layer below
// (dgrad) or an fp32 atomic add into the weight gradient (wgrad, split over K
// across CTAs).  CTAs are persistent, so tensor memory is allocated once.
//
// * dgrad: an input position takes a tap only where its parity matches, so the
//   input positions of one parity class share their 1, 2, 4 or 8 taps: one GEMM
//   per class (27 / 8 taps a position instead of 27, 7/8 of them zeros).
// * wgrad: both operands run along K in memory (positions), so they are
//   MN-major tiles, copied as they lie.  Transposed into K-major tiles two
//   bytes at a time, a chunk took ten times its loads in stores.
// * The first layer (one input channel: K = 27) gathers from a patch of the input
//   in shared memory; its weight gradient, 27 x N with the positions along K, is
//   fp32 FMAs (a lane per tap) on such a patch.
//
// Every mbarrier wait has a time limit (about 1 s of %globaltimer); a wait
// that runs out records an error code, the CTA waits (again bounded) for its
// own MMAs, frees its tensor memory and returns.
#include <algorithm>
#include <cmath>

#include <cuda_bf16.h>

#include "pmg_common.cuh"

namespace pmg {
namespace cnn {

constexpr int kBM = 128;    // tile rows = TMEM lanes
constexpr int kBK = 64;     // K elements per chunk (128 bytes of bf16)
constexpr int kStages = 3;  // shared-memory pipeline depth
constexpr int kThreads = 128;
constexpr unsigned long long kWaitNs = 1000000000ull; // 1 s

// ---- PTX wrappers -----------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long gtime()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *b, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t *b, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Bounded wait for the phase with the given parity to complete.
__device__ __forceinline__ bool mbar_wait(uint64_t *b, unsigned parity)
{
    if (mbar_try(b, parity))
        return true;
    const unsigned long long t0 = gtime();
    while (!mbar_try(b, parity))
        if (gtime() - t0 > kWaitNs)
            return false;
    return true;
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *dst, int ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, int ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// D(tmem) (+)= A(smem) * B(smem)^T, bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}

// Arrive on the mbarrier once all tcgen05 operations this thread issued
// before have completed.
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// 16 bytes global -> shared, zeros where !valid (src is then not read).
__device__ __forceinline__ void cp16(uint8_t *dst, const void *src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(valid ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 16 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v)
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++)
        v[i] = __uint_as_float(r[i]);
}

// ---- layouts and descriptors ------------------------------------------------

// Byte offset of the 16-byte chunk j (of 8) of row r in a tile stored K-major
// with the 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes
// apart, chunk index XORed with the row's position in its group.
__device__ __forceinline__ uint32_t sw128(int r, int j)
{
    return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4));
}

// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled tile
// starting at byte address addr (tile base 1024-aligned; addr may be offset
// by 32-byte K steps inside the first row): start address >> 4, leading
// byte offset 16 (unused by this layout), stride byte offset 1024 (8-row
// groups), descriptor version 1, swizzle mode 2 (128 bytes).
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// Byte offset of 16-byte chunk g (8 of the M or N index) of K index k in an
// MN-major tile of 64 K with the 128-byte swizzle: per 64 of M (N) one column
// of 8192 bytes, in it rows of 128 bytes (one k each), groups of 8 rows 1024
// bytes apart.
__device__ __forceinline__ uint32_t swmn(int k, int g)
{
    return (uint32_t)((g >> 3) * 8192 + (k >> 3) * 1024 + (k & 7) * 128 + (((g & 7) ^ (k & 7)) << 4));
}

// Descriptor of such a tile: leading byte offset 8192 (next 64 of M or N),
// stride byte offset 1024 (next 8 of K).
__device__ __forceinline__ uint64_t sdesc_mn128(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (512ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// Instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, both
// K-major or (mn, the transpose bits) both MN-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t idesc_bf16(int n, bool mn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? 3u << 15 : 0u) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(kBM >> 4) << 24);
}

// ---- convolution geometry -----------------------------------------------------

// Cubic volumes: input side di, output side do_ = (di + 1) / 2, channels-last.
struct Geo {
    int batch, di, dout, cin, cout;
    __device__ __forceinline__ long long npos_in() const { return (long long)batch * di * di * di; }
    __device__ __forceinline__ long long npos_out() const { return (long long)batch * dout * dout * dout; }
};

// ---- the three convolution operators as GEMM operand gatherers ---------------------
// (input channels >= 16; lg*: log2 of the channel counts)

// valid taps along an axis of d positions from i0 = first tap's position: bit k
__device__ __forceinline__ unsigned taps_in(int i0, int d)
{
    unsigned v = 0;
#pragma unroll
    for (int k = 0; k < 3; k++)
        v |= (unsigned)(i0 + k >= 0 && i0 + k < d) << k;
    return v;
}

// forward: rows = output positions, K = 27 * cin (tap-major), N = cout.
// B operand: Wk [cout][kp] bf16, k = tap * cin + c, zero-padded to kp.
struct OpFwd {
    static constexpr bool kMN = false;
    Geo g;
    const __nv_bfloat16 *x;  // [npos_in][cin]
    const __nv_bfloat16 *wk; // [cout][kp]
    const float *bias;       // [cout]
    __nv_bfloat16 *y;        // [npos_out][cout]
    int kp, lgc;
    FastDiv qo;
    struct Row {
        long long m, base; // base: first tap's input position
        unsigned vz, vy, vx;
    };
    __device__ __forceinline__ void chunks(int, int, int, int &kc0, int &kc1) const
    {
        kc0 = 0;
        kc1 = kp / kBK;
    }
    __device__ __forceinline__ Row row(int tile, int tid) const
    {
        Row r;
        r.m = (long long)tile * kBM + tid;
        const bool live = r.m < g.npos_out();
        const unsigned m = live ? (unsigned)r.m : 0u, q1 = fdiv(m, qo), q2 = fdiv(q1, qo), n = fdiv(q2, qo);
        const int xx = (int)(m - q1 * g.dout), yy = (int)(q1 - q2 * g.dout), z = (int)(q2 - n * g.dout), d = g.di;
        r.base = (((long long)n * d + 2 * z - 1) * d + 2 * yy - 1) * d + 2 * xx - 1;
        r.vz = live ? taps_in(2 * z - 1, d) : 0u;
        r.vy = taps_in(2 * yy - 1, d);
        r.vx = taps_in(2 * xx - 1, d);
        return r;
    }
    __device__ __forceinline__ void load(uint8_t *sa, uint8_t *sb, const Row &r, int kc, int tid, int bn) const
    {
        const int d = g.di;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k0 = kc * kBK + j * 8, t = k0 >> lgc, c0 = k0 & (g.cin - 1);
            const int kz = t / 9, ky = t / 3 - 3 * kz, kx = t - 3 * (t / 3);
            const bool in = t < 27 && ((r.vz >> kz) & (r.vy >> ky) & (r.vx >> kx) & 1u);
            cp16(sa + sw128(tid, j), in ? x + (r.base + (kz * d + ky) * d + kx) * g.cin + c0 : x, in);
        }
        for (int it = tid; it < bn * 8; it += kThreads) {
            const int o = it >> 3, j = it & 7;
            cp16(sb + sw128(o, j), wk + (long long)o * kp + kc * kBK + j * 8, true);
        }
    }
    __device__ __forceinline__ void store(const Row &r, int c0, const float *v) const
    {
        if (r.m >= g.npos_out())
            return;
        __align__(16) __nv_bfloat16 o[16];
#pragma unroll
        for (int i = 0; i < 16; i++)
            o[i] = __float2bfloat16(fmaxf(v[i] + bias[c0 + i], 0.0f));
        uint4 *dst = reinterpret_cast<uint4 *>(y + r.m * g.cout + c0);
        dst[0] = reinterpret_cast<const uint4 *>(o)[0];
        dst[1] = reinterpret_cast<const uint4 *>(o)[1];
    }
};

// dgrad: rows = input positions of one parity class, K = its taps * cout, N =
// cin.  Input iz takes tap kz from output oz when iz = 2 oz + kz - 1: an even
// one tap 1 from iz / 2, an odd one tap 0 from (iz + 1) / 2 and tap 2 from
// (iz - 1) / 2.  B operand: WkT [cin][kp] bf16, k = tap * cout + o.  The result
// is masked by ReLU' of the layer below (its output xact > 0) -- the gradient of
// that layer's pre-activation.
struct OpDgrad {
    static constexpr bool kMN = false;
    Geo g;
    const __nv_bfloat16 *dz;   // [npos_out][cout]
    const __nv_bfloat16 *wkt;  // [cin][kp]
    const __nv_bfloat16 *xact; // [npos_in][cin]
    __nv_bfloat16 *dx;         // [npos_in][cin]
    int kp, lgc;
    int first[9];         // first tile of each class, the most taps first
    FastDiv qh[2];        // division by the even and the odd positions of an axis
    int nh[2];
    struct Row {
        long long pos;     // input position, -1: none
        long long base;    // output position (n, a, b, c)
        int cls;           // odd axes: bits 2 (z), 1 (y), 0 (x)
        unsigned hz, hy, hx; // the next output of an odd axis exists
    };
    __device__ __forceinline__ int cls_of(int tile) const
    {
        int c = 0;
#pragma unroll
        for (int k = 1; k < 8; k++)
            c += tile >= first[k];
        return 7 - c;
    }
    __device__ __forceinline__ void chunks(int tile, int, int, int &kc0, int &kc1) const
    {
        kc0 = 0;
        kc1 = ((g.cout << __popc(cls_of(tile))) + kBK - 1) / kBK;
    }
    __device__ __forceinline__ Row row(int tile, int tid) const
    {
        Row r;
        r.cls = cls_of(tile);
        const int pz = r.cls >> 2, py = (r.cls >> 1) & 1, px = r.cls & 1;
        const unsigned nz = nh[pz], ny = nh[py], nx = nh[px];
        const unsigned m = (unsigned)((tile - first[7 - r.cls]) * kBM + tid), rows = g.batch * nz * ny * nx;
        const unsigned q1 = fdiv(m, qh[px]), q2 = fdiv(q1, qh[py]), n = fdiv(q2, qh[pz]);
        const int c = (int)(m - q1 * nx), b = (int)(q1 - q2 * ny), a = (int)(q2 - n * nz);
        r.pos = m < rows ? (((long long)n * g.di + 2 * a + pz) * g.di + 2 * b + py) * g.di + 2 * c + px : -1;
        r.base = (((long long)n * g.dout + a) * g.dout + b) * g.dout + c;
        r.hz = a + 1 < g.dout;
        r.hy = b + 1 < g.dout;
        r.hx = c + 1 < g.dout;
        return r;
    }
    __device__ __forceinline__ void load(uint8_t *sa, uint8_t *sb, const Row &r, int kc, int tid, int bn) const
    {
        const int pz = r.cls >> 2, py = (r.cls >> 1) & 1, px = r.cls & 1, ntaps = 1 << __popc(r.cls), d = g.dout;
        // local tap t: one bit per odd axis, 0: tap 0 (the next output), 1: tap 2
        auto bits = [&](int t, int &bz, int &by, int &bx) {
            bx = px ? t & 1 : 1;
            t >>= px;
            by = py ? t & 1 : 1;
            t >>= py;
            bz = pz ? t & 1 : 1;
        };
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k0 = kc * kBK + j * 8, t = k0 >> lgc, o0 = k0 & (g.cout - 1);
            int bz, by, bx;
            bits(t, bz, by, bx);
            const bool in = t < ntaps && r.pos >= 0 && (bz || r.hz) && (by || r.hy) && (bx || r.hx);
            cp16(sa + sw128(tid, j), in ? dz + (r.base + ((1 - bz) * d + 1 - by) * d + 1 - bx) * g.cout + o0 : dz, in);
        }
        for (int it = tid; it < bn * 8; it += kThreads) {
            const int c = it >> 3, j = it & 7, k0 = kc * kBK + j * 8, t = k0 >> lgc, o0 = k0 & (g.cout - 1);
            int bz, by, bx;
            bits(t, bz, by, bx);
            const int tap = ((pz ? 2 * bz : 1) * 3 + (py ? 2 * by : 1)) * 3 + (px ? 2 * bx : 1);
            cp16(sb + sw128(c, j), t < ntaps ? wkt + (long long)c * kp + tap * g.cout + o0 : wkt, t < ntaps);
        }
    }
    __device__ __forceinline__ void store(const Row &r, int c0, const float *v) const
    {
        if (r.pos < 0)
            return;
        const uint4 *xa = reinterpret_cast<const uint4 *>(xact + r.pos * g.cin + c0);
        __align__(16) __nv_bfloat16 x[16], o[16];
        reinterpret_cast<uint4 *>(x)[0] = xa[0];
        reinterpret_cast<uint4 *>(x)[1] = xa[1];
#pragma unroll
        for (int i = 0; i < 16; i++)
            o[i] = __float2bfloat16(__bfloat162float(x[i]) > 0.0f ? v[i] : 0.0f);
        uint4 *dst = reinterpret_cast<uint4 *>(dx + r.pos * g.cin + c0);
        dst[0] = reinterpret_cast<const uint4 *>(o)[0];
        dst[1] = reinterpret_cast<const uint4 *>(o)[1];
    }
};

// wgrad: rows = (tap, c_in) pairs (27 * cin, tile rows beyond are zero), K =
// output positions (split over CTAs), N = 64 (columns beyond cout are zero).
// The result is added into dw [27 * cin][cout] fp32 with atomics.
struct OpWgrad {
    static constexpr bool kMN = true;
    Geo g;
    const __nv_bfloat16 *x;  // [npos_in][cin]
    const __nv_bfloat16 *dz; // [npos_out][cout]
    float *dw;               // [27 * cin][cout]
    int kchunks_total;       // ceil(npos_out / 64)
    int lgc;
    int vec;                 // dw is 16-byte aligned
    FastDiv qo;
    struct Row {
        int m;                // this thread's accumulator row
        int kz, ky, kx, c0;   // of the eight rows that it gathers (kz < 0: none)
    };
    __device__ __forceinline__ void chunks(int, int split, int nsplit, int &kc0, int &kc1) const
    {
        const int per = (kchunks_total + nsplit - 1) / nsplit;
        kc0 = split * per;
        kc1 = min(kchunks_total, kc0 + per);
    }
    __device__ __forceinline__ Row row(int tile, int tid) const
    {
        Row r;
        r.m = tile * kBM + tid;
        const int r0 = tile * kBM + (tid & 15) * 8, t = r0 >> lgc;
        r.c0 = r0 & (g.cin - 1);
        r.kz = t < 27 ? t / 9 : -1;
        r.ky = t / 3 % 3;
        r.kx = t % 3;
        return r;
    }
    __device__ __forceinline__ void load(uint8_t *sa, uint8_t *sb, const Row &r, int kc, int tid, int) const
    {
        const unsigned np = (unsigned)g.npos_out();
        const int d = g.di, dd = g.dout;
        // A: 64 positions x 16 groups of 8 rows; this thread group tid % 16
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int j = (tid >> 4) + 8 * u;
            const unsigned p = (unsigned)kc * kBK + j, q1 = fdiv(p, qo), q2 = fdiv(q1, qo), n = fdiv(q2, qo);
            const int iz = 2 * (int)(q2 - n * dd) + r.kz - 1, iy = 2 * (int)(q1 - q2 * dd) + r.ky - 1,
                      ix = 2 * (int)(p - q1 * dd) + r.kx - 1;
            const bool in = r.kz >= 0 && p < np && iz >= 0 && iz < d && iy >= 0 && iy < d && ix >= 0 && ix < d;
            cp16(sa + swmn(j, tid & 15), in ? x + ((((long long)n * d + iz) * d + iy) * d + ix) * g.cin + r.c0 : x, in);
        }
        // B: 64 positions x 8 groups of 8 columns
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int j = (tid >> 3) + 16 * u, c0 = (tid & 7) * 8;
            const unsigned p = (unsigned)kc * kBK + j;
            const bool in = p < np && c0 < g.cout;
            cp16(sb + swmn(j, tid & 7), in ? dz + (long long)p * g.cout + c0 : dz, in);
        }
    }
    __device__ __forceinline__ void store(const Row &r, int c0, const float *v) const
    {
        if (r.m >= 27 * g.cin || c0 >= g.cout)
            return;
        float *dst = dw + (long long)r.m * g.cout + c0;
        if (vec) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                atomicAdd(reinterpret_cast<float4 *>(dst) + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++)
                atomicAdd(dst + i, v[i]);
        }
    }
};

// ---- the tile kernel ----------------------------------------------------------------

template <int BN>
struct TileSmem {
    static constexpr int kA = kBM * 128; // 16 KB per A stage
    static constexpr int kB = BN * 128;  // B stage
    static constexpr int kStage = kA + kB;
    static constexpr int kBytes = kStages * kStage + 1024; // + alignment slack
};

// Error codes written to *err: 1 = an mbarrier wait ran out of time.
// Bound by the gather's latency and L2 traffic (a chunk's 16 to 24 KB are a few
// hundred cycles of tensor core work), hence two chunks in flight per CTA and
// three to four CTAs on an SM.  At batch 64, three layers: forward 0.15, dgrad
// 0.21, wgrad 0.13 ms; with loads that each chunk waited for, K-major wgrad tiles
// and all 27 taps in dgrad, four layers took 0.67, 1.51 and 1.14 ms.
template <class Op, int BN>
__global__ void __launch_bounds__(kThreads) k_umma_conv(Op op, int ntiles, int ksplit, int *err)
{
    static_assert(BN == 16 || BN == 32 || BN == 64, "tile width");
    constexpr int kCols = BN < 32 ? 32 : BN; // TMEM allocation: a power of two >= 32
    constexpr uint32_t kIdesc = idesc_bf16(BN, Op::kMN);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar[kStages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_base;

    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5;

    if (warp == 0) {
        tmem_alloc(&tmem_base, kCols);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < kStages; s++)
            mbar_init(&bar[s], 1);
        mbar_init(&done_bar, 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;

    bool ok = true;
    int gi = 0; // chunks of the earlier items: chunk i of this one is use (gi + i) / kStages of its stage
    const int items = ntiles * ksplit;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int tile = item / ksplit;
        int kc0, kc1;
        op.chunks(tile, item - tile * ksplit, ksplit, kc0, kc1);
        const int n = kc1 - kc0;
        if (n <= 0)
            continue;
        const typename Op::Row row = op.row(tile, tid);
        // chunk i into its stage, once the MMAs of the stage's last use are done
        auto fetch = [&](int i) {
            if (i < n) {
                const int use = gi + i, s = use % kStages;
                if (use >= kStages)
                    ok = mbar_wait(&bar[s], (unsigned)(use / kStages - 1) & 1u) && ok;
                uint8_t *sa = smem + s * TileSmem<BN>::kStage;
                if (ok)
                    op.load(sa, sa + TileSmem<BN>::kA, row, kc0 + i, tid, BN);
            }
            cp_commit(); // (a group per chunk, empty past the last)
        };
        fetch(0);
        fetch(1);
        int i = 0;
        for (; i < n; i++) {
            cp_wait<1>(); // chunk i has landed
            fence_async_smem();
            if (!__syncthreads_and(ok)) {
                ok = false;
                break;
            }
            if (tid == 0) {
                tc_fence_after();
                const int s = (gi + i) % kStages;
                const uint32_t a0 = smem_u32(smem + s * TileSmem<BN>::kStage), b0 = a0 + TileSmem<BN>::kA;
#pragma unroll
                for (int kk = 0; kk < kBK / 16; kk++)
                    umma_bf16(tmem, Op::kMN ? sdesc_mn128(a0 + kk * 2048) : sdesc_sw128(a0 + kk * 32),
                              Op::kMN ? sdesc_mn128(b0 + kk * 2048) : sdesc_sw128(b0 + kk * 32), kIdesc,
                              (i > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&bar[s]);
            }
            fetch(i + 2);
        }
        if (!ok)
            break;
        gi += n;
        // the item's last MMA (and so all of them)
        ok = mbar_wait(&bar[(gi - 1) % kStages], (unsigned)((gi - 1) / kStages) & 1u);
        tc_fence_after();
        // one decision for the whole CTA: tcgen05.ld below is warp-collective
        ok = __syncthreads_and(ok) != 0;
        if (ok) {
            const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float v[16];
                tmem_ld16(lane_addr + (uint32_t)c0, v);
                op.store(row, c0, v);
            }
        }
        // the next item's MMAs overwrite the accumulator
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }
    cp_wait<0>();
    if (!__syncthreads_and(ok)) {
        // own MMAs in flight, for a bounded time
        if (tid == 0) {
            atomicExch(err, 1);
            umma_commit(&done_bar);
        }
        mbar_wait(&done_bar, 0);
        tc_fence_after();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        tmem_dealloc(tmem, kCols);
}

template <class Op, int BN>
static int launch_tiles(const Op &op, int ntiles, int ksplit, int *err, cudaStream_t st, const char *name,
                        double flops)
{
    const int smem = TileSmem<BN>::kBytes;
    PMG_CUDA(cudaFuncSetAttribute(k_umma_conv<Op, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    // resident CTAs: shared memory (227 KB of an SM) allows three or four
    const long long items = (long long)ntiles * ksplit;
    const unsigned grid = (unsigned)std::min<long long>(items, 152LL * (227 * 1024 / (smem + 1024)));
    const int ps__ = prof_begin(name, st);
    k_umma_conv<Op, BN><<<grid, kThreads, smem, st>>>(op, ntiles, ksplit, err);
    prof_end(ps__, flops, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

template <class Op>
static int launch_bn(const Op &op, int bn, int ntiles, int ksplit, int *err, cudaStream_t st, const char *name,
                     double flops)
{
    switch (bn) {
    case 16:
        return launch_tiles<Op, 16>(op, ntiles, ksplit, err, st, name, flops);
    case 32:
        return launch_tiles<Op, 32>(op, ntiles, ksplit, err, st, name, flops);
    case 64:
        return launch_tiles<Op, 64>(op, ntiles, ksplit, err, st, name, flops);
    default:
        set_error("cnn: output channels %d not in {16, 32, 64}", bn);
        return PMG_EINVAL;
    }
}

// ---- the first layer: one input channel ---------------------------------------------
constexpr int kPatchX = 32, kPatchY = 4; // output positions of a tile: 128

// Forward: the tile kernel's GEMM with the A rows built from the patch of the
// input that the 4 x 32 positions read (even and odd columns apart, so that a
// warp's reads are consecutive).  K is 27 padded to 32; a GEMM over the 64 that
// the weights are padded to adds zeros.  Bound by the patch's loads and the 32
// bytes written per position; taps gathered one by one from global memory were
// most of the forward's 0.67 ms at batch 64, this is 0.08 ms.
template <int BN>
__global__ void __launch_bounds__(kThreads) k_conv1_fwd(const __nv_bfloat16 *__restrict__ x,
                                                        const __nv_bfloat16 *__restrict__ wk, int kp,
                                                        const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y,
                                                        int d, int dd, int ty, int tx, int ntiles, int *err)
{
    constexpr int kCols = BN < 32 ? 32 : BN, kRows = 2 * kPatchY + 1;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __nv_bfloat16 s_e[3][kRows][kPatchX + 2], s_o[3][kRows][kPatchX];
    __shared__ __align__(8) uint64_t bar, done_bar;
    __shared__ uint32_t tmem_base;
    uint8_t *sa = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *sb = sa + kBM * 128;
    const int tid = threadIdx.x, warp = tid >> 5, xl = tid & 31, yl = tid >> 5;
    if (warp == 0) {
        tmem_alloc(&tmem_base, kCols);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_init(&done_bar, 1);
        fence_barrier_init();
    }
    for (int it = tid; it < BN * 4; it += kThreads) {
        const int r = it >> 2, j = it & 3;
        *reinterpret_cast<uint4 *>(sb + sw128(r, j)) =
            *reinterpret_cast<const uint4 *>(wk + (long long)r * kp + j * 8);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    unsigned phase = 0;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        int t = tile;
        const int xb = t % tx;
        t /= tx;
        const int yb = t % ty;
        t /= ty;
        const int z = t % dd, n = t / dd;
        // patch column c is input column ix0 - 1 + c: pairs (2 q + 1, 2 q + 2) from input column ix0 + 2 q
        const int ix0 = 2 * xb * kPatchX, iy0 = 2 * yb * kPatchY - 1;
        for (int it = tid; it < 3 * kRows * (kPatchX + 1); it += kThreads) {
            const int row = it / (kPatchX + 1), q = it - row * (kPatchX + 1) - 1;
            const int kz = row / kRows, yy = row - kz * kRows;
            const int iz = 2 * z - 1 + kz, iy = iy0 + yy, ix = ix0 + 2 * q;
            __nv_bfloat16 a = __float2bfloat16(0.0f), b = a;
            if (iz >= 0 && iz < d && iy >= 0 && iy < d) {
                const __nv_bfloat16 *src = x + (((long long)n * d + iz) * d + iy) * d;
                if (ix >= 0 && ix < d)
                    a = src[ix];
                if (ix + 1 >= 0 && ix + 1 < d)
                    b = src[ix + 1];
            }
            if (q >= 0)
                s_o[kz][yy][q] = a;
            s_e[kz][yy][q + 1] = b;
        }
        __syncthreads();
        __align__(16) __nv_bfloat16 k[32];
#pragma unroll
        for (int tap = 0; tap < 32; tap++) {
            const int kz = tap / 9, ky = tap / 3 % 3, kx = tap % 3;
            if (tap < 27)
                k[tap] = kx == 1 ? s_o[kz][2 * yl + ky][xl] : s_e[kz][2 * yl + ky][xl + (kx >> 1)];
            else
                k[tap] = __float2bfloat16(0.0f);
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            *reinterpret_cast<uint4 *>(sa + sw128(tid, j)) = reinterpret_cast<const uint4 *>(k)[j];
        fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sb);
#pragma unroll
            for (int kk = 0; kk < 2; kk++)
                umma_bf16(tmem, sdesc_sw128(a0 + kk * 32), sdesc_sw128(b0 + kk * 32), idesc_bf16(BN, false), kk > 0);
            umma_commit(&bar);
        }
        ok = mbar_wait(&bar, phase);
        phase ^= 1u;
        tc_fence_after();
        ok = __syncthreads_and(ok) != 0; // tcgen05.ld is warp-collective
        if (ok) {
            const int ox = xb * kPatchX + xl, oy = yb * kPatchY + yl;
            const bool in = ox < dd && oy < dd;
            __nv_bfloat16 *dst = y + ((((long long)n * dd + z) * dd + oy) * dd + ox) * BN;
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
                __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                for (int c = 0; c < 16; c++)
                    o[c] = __float2bfloat16(fmaxf(v[c] + bias[c0 + c], 0.0f));
                if (in) {
                    reinterpret_cast<uint4 *>(dst + c0)[0] = reinterpret_cast<const uint4 *>(o)[0];
                    reinterpret_cast<uint4 *>(dst + c0)[1] = reinterpret_cast<const uint4 *>(o)[1];
                }
            }
        }
        tc_fence_before(); // (the next MMA overwrites the accumulator, after two barriers)
    }
    if (!__syncthreads_and(ok)) {
        if (tid == 0) {
            atomicExch(err, 1);
            umma_commit(&done_bar);
        }
        mbar_wait(&done_bar, 0);
        tc_fence_after();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        tmem_dealloc(tmem, kCols);
}

static int kpad(int k) { return (k + kBK - 1) / kBK * kBK; }

template <int BN>
static int launch_conv1_fwd(const __nv_bfloat16 *x, const __nv_bfloat16 *wk, const float *bias, __nv_bfloat16 *y,
                            const Geo &g, int *err, cudaStream_t st)
{
    const int smem = kBM * 128 + BN * 128 + 1024;
    PMG_CUDA(cudaFuncSetAttribute(k_conv1_fwd<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int ty = (g.dout + kPatchY - 1) / kPatchY, tx = (g.dout + kPatchX - 1) / kPatchX;
    const long long tiles = (long long)g.batch * g.dout * ty * tx;
    const int ps__ = prof_begin("k_conv1_fwd", st);
    k_conv1_fwd<BN><<<(unsigned)std::min<long long>(tiles, 152 * 8), kThreads, smem, st>>>(
        x, wk, kpad(27), bias, y, g.di, g.dout, ty, tx, (int)tiles, err);
    prof_end(ps__, 2.0 * g.batch * g.dout * g.dout * g.dout * g.cout * 27.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// Weight gradient: a warp takes 32 output positions of a row one after the
// other, lane = tap (lane 27: the constant 1, whose row is the bias gradient),
// 16 output channels (blockIdx.y) in registers.  128 threads on 4 x 32 positions,
// blocks stride over the tiles.  Bound by the shared-memory reads that feed the
// FMAs and by the patch's loads: 0.15 ms at batch 64.
constexpr int kWgY = 4;

__global__ void __launch_bounds__(128) k_conv1_wgrad(const __nv_bfloat16 *__restrict__ x,
                                                     const __nv_bfloat16 *__restrict__ dz, float *__restrict__ dw,
                                                     float *__restrict__ db, int d, int dd, int cout, int ty, int tx,
                                                     int ntiles)
{
    // banks of the 27 taps of one position: row stride 67 = 3, plane stride 617 = 9 (mod 32)
    constexpr int kRows = 2 * kWgY + 1, kCols = 2 * kPatchX + 1, kRS = 67, kPS = 617;
    static_assert(kRows * kRS <= kPS, "planes do not overlap");
    __shared__ float s_x[3 * kPS];
    __shared__ __align__(16) float s_d[128][16];
    const int c0 = blockIdx.y * 16, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int kz = lane / 9, ky = lane / 3 % 3, kx = lane % 3;
    const float fixed = lane == 27 ? 1.0f : 0.0f;
    float acc[16];
#pragma unroll
    for (int c = 0; c < 16; c++)
        acc[c] = 0.0f;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int t = tile;
        const int xb = t % tx;
        t /= tx;
        const int yb = t % ty;
        t /= ty;
        const int z = t % dd, n = t / dd;
        __syncthreads(); // (the last tile's readers)
        for (int it = threadIdx.x; it < 3 * kRows * kCols; it += blockDim.x) {
            const int row = it / kCols, c = it - row * kCols, pz = row / kRows, yy = row - pz * kRows;
            const int iz = 2 * z - 1 + pz, iy = 2 * yb * kWgY - 1 + yy, ix = 2 * xb * kPatchX - 1 + c;
            const bool in = iz >= 0 && iz < d && iy >= 0 && iy < d && ix >= 0 && ix < d;
            s_x[pz * kPS + yy * kRS + c] =
                in ? __bfloat162float(x[(((long long)n * d + iz) * d + iy) * d + ix]) : 0.0f;
        }
        {
            const int oy = yb * kWgY + w, ox = xb * kPatchX + lane;
            uint4 q[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
            if (oy < dd && ox < dd) {
                const uint4 *src =
                    reinterpret_cast<const uint4 *>(dz + ((((long long)n * dd + z) * dd + oy) * dd + ox) * cout + c0);
                q[0] = src[0];
                q[1] = src[1];
            }
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(q);
            float4 *dst = reinterpret_cast<float4 *>(s_d[threadIdx.x]);
#pragma unroll
            for (int c = 0; c < 4; c++)
                dst[c] = make_float4(__bfloat162float(e[4 * c]), __bfloat162float(e[4 * c + 1]),
                                     __bfloat162float(e[4 * c + 2]), __bfloat162float(e[4 * c + 3]));
        }
        __syncthreads();
        const float *sx = s_x + (lane < 27 ? kz * kPS + (2 * w + ky) * kRS + kx : 0);
        // (only the positions inside: beyond them an input may still be read, and a
        // zero gradient times one that is not finite is not zero)
        const int np = yb * kWgY + w < dd ? min(32, dd - xb * kPatchX) : 0;
#pragma unroll 4
        for (int p = 0; p < np; p++) {
            const float v = lane < 27 ? sx[2 * p] : fixed;
            const float4 *q = reinterpret_cast<const float4 *>(s_d[w * 32 + p]);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float4 f = q[c];
                acc[4 * c] = __fmaf_rn(v, f.x, acc[4 * c]);
                acc[4 * c + 1] = __fmaf_rn(v, f.y, acc[4 * c + 1]);
                acc[4 * c + 2] = __fmaf_rn(v, f.z, acc[4 * c + 2]);
                acc[4 * c + 3] = __fmaf_rn(v, f.w, acc[4 * c + 3]);
            }
        }
    }
    // the four warps' sums, then one add per block
    __syncthreads();
    float4 *mine = reinterpret_cast<float4 *>(s_d[threadIdx.x]);
#pragma unroll
    for (int c = 0; c < 4; c++)
        mine[c] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
    __syncthreads();
    for (int it = threadIdx.x; it < 28 * 16; it += blockDim.x) {
        const int tap = it >> 4, c = it & 15;
        const float v = s_d[tap][c] + s_d[32 + tap][c] + s_d[64 + tap][c] + s_d[96 + tap][c];
        atomicAdd(tap < 27 ? dw + tap * cout + c0 + c : db + c0 + c, v);
    }
}

static int check_geo(int batch, int di, int cin, int cout)
{
    if (batch <= 0 || di <= 1 || di > 1024) {
        set_error("cnn: batch %d / side %d out of range", batch, di);
        return PMG_EINVAL;
    }
    if (!(cin == 1 || cin == 16 || cin == 32 || cin == 64) || !(cout == 16 || cout == 32 || cout == 64)) {
        set_error("cnn: channels %d -> %d not supported (cin in {1,16,32,64}, cout in {16,32,64})", cin, cout);
        return PMG_EINVAL;
    }
    return PMG_OK;
}


static int log2_of(int c) { return c == 16 ? 4 : c == 32 ? 5 : 6; }

// ---- weight packing (fp32 master [cout][cin][27] -> bf16 GEMM operands) -------------

__global__ void k_pack_w(const float *__restrict__ w, int cin, int cout, int kp, __nv_bfloat16 *__restrict__ wk,
                         int kpt, __nv_bfloat16 *__restrict__ wkt)
{
    const int n1 = cout * kp, n2 = wkt ? cin * kpt : 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n1 + n2; i += gridDim.x * blockDim.x) {
        if (i < n1) {
            const int o = i / kp, k = i - o * kp;
            const int t = k / cin, c = k - t * cin;
            wk[i] = __float2bfloat16(t < 27 ? w[((long long)o * cin + c) * 27 + t] : 0.0f);
        } else {
            const int i2 = i - n1;
            const int c = i2 / kpt, k = i2 - c * kpt;
            const int t = k / cout, o = k - t * cout;
            wkt[i2] = __float2bfloat16(t < 27 ? w[((long long)o * cin + c) * 27 + t] : 0.0f);
        }
    }
}

// dw [27 * cin][cout] (tap-major rows) -> grad [cout][cin][27]
__global__ void k_unpack_dw(const float *__restrict__ dw, int cin, int cout, float *__restrict__ grad)
{
    const int n = cout * cin * 27;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int t = i % 27, c = (i / 27) % cin, o = i / (27 * cin);
        grad[i] = dw[((long long)t * cin + c) * cout + o];
    }
}

// bias gradient: db[o] = sum over positions of dz[p][o]; eight channels per
// thread.
__global__ void __launch_bounds__(256) k_bias_grad(const __nv_bfloat16 *__restrict__ dz, long long np, int cout,
                                                   float *__restrict__ db)
{
    __shared__ float acc[64];
    if (threadIdx.x < 64)
        acc[threadIdx.x] = 0.0f;
    __syncthreads();
    const int groups = cout >> 3, gr = threadIdx.x % groups, lanes = blockDim.x / groups;
    float s[8] = {};
    for (long long p = (long long)blockIdx.x * lanes + threadIdx.x / groups; p < np; p += (long long)gridDim.x * lanes) {
        const uint4 v = *reinterpret_cast<const uint4 *>(dz + p * cout + gr * 8);
        const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
        for (int i = 0; i < 8; i++)
            s[i] += __bfloat162float(e[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; i++)
        atomicAdd(&acc[gr * 8 + i], s[i]);
    __syncthreads();
    if (threadIdx.x < cout)
        atomicAdd(db + threadIdx.x, acc[threadIdx.x]);
}

// ---- head: global average pool, MLP 64-64-64, sigmoid, MSE loss and its backward ----
// One CTA of 64 threads per sample.  y4: [batch][64 positions][64 channels]
// bf16 (the last convolution's ReLU output, 4^3 positions); parameters fp32:
// w5 [64][64] b5 [64] (hidden, ReLU), w6 [64][64] b6 [64] (outputs, sigmoid).
// With target != null the loss mean((s - t)^2) / batch is accumulated into
// *loss and the gradients are added into the g* buffers (atomics across
// samples) and written to dy4 (masked by the last ReLU).
constexpr int kHead = 64;

__global__ void k_head(const __nv_bfloat16 *__restrict__ y4, const float *__restrict__ w5,
                       const float *__restrict__ b5, const float *__restrict__ w6, const float *__restrict__ b6,
                       const float *__restrict__ target, float *__restrict__ pred, float *__restrict__ loss,
                       float *__restrict__ gw5, float *__restrict__ gb5, float *__restrict__ gw6,
                       float *__restrict__ gb6, __nv_bfloat16 *__restrict__ dy4, float inv_batch)
{
    __shared__ float h0[kHead], h1[kHead], dout[kHead], dh1[kHead];
    const int n = blockIdx.x, t = threadIdx.x;
    const __nv_bfloat16 *y = y4 + (long long)n * 64 * kHead;
    float a = 0.0f;
    for (int p = 0; p < 64; p++)
        a += __bfloat162float(y[p * kHead + t]);
    h0[t] = a * (1.0f / 64.0f);
    __syncthreads();
    float z = b5[t];
    for (int c = 0; c < kHead; c++)
        z += w5[t * kHead + c] * h0[c];
    h1[t] = fmaxf(z, 0.0f);
    __syncthreads();
    float o = b6[t];
    for (int j = 0; j < kHead; j++)
        o += w6[t * kHead + j] * h1[j];
    const float s = 1.0f / (1.0f + __expf(-o));
    pred[(long long)n * kHead + t] = s;
    if (!target)
        return;
    const float e = s - target[(long long)n * kHead + t];
    atomicAdd(loss, e * e * (inv_batch / kHead));
    dout[t] = 2.0f * e * (inv_batch / kHead) * s * (1.0f - s);
    __syncthreads();
    for (int j = 0; j < kHead; j++)
        atomicAdd(gw6 + t * kHead + j, dout[t] * h1[j]);
    atomicAdd(gb6 + t, dout[t]);
    float d1 = 0.0f;
    for (int k = 0; k < kHead; k++)
        d1 += w6[k * kHead + t] * dout[k];
    dh1[t] = h1[t] > 0.0f ? d1 : 0.0f;
    __syncthreads();
    for (int c = 0; c < kHead; c++)
        atomicAdd(gw5 + t * kHead + c, dh1[t] * h0[c]);
    atomicAdd(gb5 + t, dh1[t]);
    float d0 = 0.0f;
    for (int j = 0; j < kHead; j++)
        d0 += w5[j * kHead + t] * dh1[j];
    d0 *= 1.0f / 64.0f;
    __nv_bfloat16 *dy = dy4 + (long long)n * 64 * kHead;
    for (int p = 0; p < 64; p++)
        dy[p * kHead + t] = __float2bfloat16(__bfloat162float(y[p * kHead + t]) > 0.0f ? d0 : 0.0f);
}

// Adam (Kingma and Ba) over a flat fp32 parameter vector, bias-corrected.
__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, long long n, float lr, float b1, float b2, float eps, float c1,
                       float c2, float wd)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i] + wd * w[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// Network input: the distance field of the own region, averaged over 64^3
// cells (cell a of an axis of length L covers [a L / 64, (a + 1) L / 64)),
// divided by `scale` (the medium's largest distance), as bf16.
__global__ void k_downsample(const float *__restrict__ d, long long s1, long long s2, int lo0, int lo1, int lo2,
                             int l0, int l1, int l2, float inv_scale, __nv_bfloat16 *__restrict__ out)
{
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= 64 * 64 * 64)
        return;
    const int a = cell >> 12, b = (cell >> 6) & 63, c = cell & 63;
    const int i0 = a * l0 / 64, i1 = (a + 1) * l0 / 64;
    const int j0 = b * l1 / 64, j1 = (b + 1) * l1 / 64;
    const int k0 = c * l2 / 64, k1 = (c + 1) * l2 / 64;
    float acc = 0.0f;
    int cnt = 0;
    for (int i = i0; i < i1; i++)
        for (int j = j0; j < j1; j++)
            for (int k = k0; k < k1; k++) {
                acc += d[((long long)(lo0 + i) * s1 + (lo1 + j)) * s2 + (lo2 + k)];
                cnt++;
            }
    out[cell] = __float2bfloat16(cnt ? acc / cnt * inv_scale : 0.0f);
}

} // namespace cnn
} // namespace pmg

using namespace pmg;
using namespace pmg::cnn;

namespace {
int cnn_err_check(int *err, cudaStream_t st)
{
    int h = 0;
    PMG_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    PMG_CUDA(cudaStreamSynchronize(st));
    if (h) {
        set_error("cnn: a tensor-core pipeline wait ran out of time (code %d)", h);
        return PMG_EITER;
    }
    return PMG_OK;
}
} // namespace

extern "C" int pmg_cnn_pack_weights(const float *w, int32_t cin, int32_t cout, void *wk, void *wkt, void *stream)
{
    if (!w || !wk) {
        set_error("pmg_cnn_pack_weights: null argument");
        return PMG_EINVAL;
    }
    const int kp = kpad(27 * cin), kpt = kpad(27 * cout);
    cudaStream_t st = as_stream(stream);
    const int ps__ = prof_begin("k_pack_w", st);
    k_pack_w<<<64, 256, 0, st>>>(w, cin, cout, kp, (__nv_bfloat16 *)wk, kpt, (__nv_bfloat16 *)wkt);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

extern "C" int pmg_cnn_conv_fwd(const void *x, const void *wk, const float *bias, void *y, int32_t batch,
                                int32_t di, int32_t cin, int32_t cout, int32_t *err, void *stream)
{
    if (!x || !wk || !bias || !y || !err) {
        set_error("pmg_cnn_conv_fwd: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_geo(batch, di, cin, cout));
    cudaStream_t st = as_stream(stream);
    const Geo g{batch, di, (di + 1) / 2, cin, cout};
    const long long rows = (long long)batch * g.dout * g.dout * g.dout;
    if (cin == 1) {
        const auto *px = (const __nv_bfloat16 *)x, *pw = (const __nv_bfloat16 *)wk;
        auto *py = (__nv_bfloat16 *)y;
        return cout == 16   ? launch_conv1_fwd<16>(px, pw, bias, py, g, err, st)
               : cout == 32 ? launch_conv1_fwd<32>(px, pw, bias, py, g, err, st)
                            : launch_conv1_fwd<64>(px, pw, bias, py, g, err, st);
    }
    OpFwd op;
    op.g = g;
    op.x = (const __nv_bfloat16 *)x;
    op.wk = (const __nv_bfloat16 *)wk;
    op.bias = bias;
    op.y = (__nv_bfloat16 *)y;
    op.kp = kpad(27 * cin);
    op.lgc = log2_of(cin);
    op.qo = fastdiv_of((unsigned)g.dout);
    return launch_bn(op, cout, (int)((rows + kBM - 1) / kBM), 1, err, st, "k_umma_conv_fwd",
                     2.0 * rows * cout * 27.0 * cin);
}

extern "C" int pmg_cnn_conv_dgrad(const void *dz, const void *wkt, const void *xact, void *dx, int32_t batch,
                                  int32_t di, int32_t cin, int32_t cout, int32_t *err, void *stream)
{
    if (!dz || !wkt || !xact || !dx || !err) {
        set_error("pmg_cnn_conv_dgrad: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_geo(batch, di, cin, cout));
    if (cin < 16) {
        set_error("pmg_cnn_conv_dgrad: the input gradient of a %d-channel layer is not needed", cin);
        return PMG_EINVAL;
    }
    OpDgrad op;
    op.g = Geo{batch, di, (di + 1) / 2, cin, cout};
    op.dz = (const __nv_bfloat16 *)dz;
    op.wkt = (const __nv_bfloat16 *)wkt;
    op.xact = (const __nv_bfloat16 *)xact;
    op.dx = (__nv_bfloat16 *)dx;
    op.kp = kpad(27 * cout);
    op.lgc = log2_of(cout);
    op.nh[0] = (di + 1) / 2;
    op.nh[1] = di / 2;
    for (int p = 0; p < 2; p++)
        op.qh[p] = fastdiv_of((unsigned)op.nh[p]);
    long long tiles = 0;
    for (int k = 0; k < 8; k++) {
        const int c = 7 - k;
        op.first[k] = (int)tiles;
        tiles += ((long long)batch * op.nh[c >> 2] * op.nh[(c >> 1) & 1] * op.nh[c & 1] + kBM - 1) / kBM;
    }
    op.first[8] = (int)tiles;
    const long long rows = (long long)batch * di * di * di;
    return launch_bn(op, cin, (int)tiles, 1, err, as_stream(stream), "k_umma_conv_dgrad",
                     2.0 * rows * cin * 27.0 * cout / 8.0);
}

extern "C" int pmg_cnn_conv_wgrad(const void *x, const void *dz, float *dw, float *grad, float *dbias,
                                  int32_t batch, int32_t di, int32_t cin, int32_t cout, int32_t *err,
                                  void *stream)
{
    if (!x || !dz || !dw || !grad || !dbias || !err) {
        set_error("pmg_cnn_conv_wgrad: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_geo(batch, di, cin, cout));
    cudaStream_t st = as_stream(stream);
    const Geo g{batch, di, (di + 1) / 2, cin, cout};
    const long long np = (long long)batch * g.dout * g.dout * g.dout;
    const long long rows = 27LL * cin;
    PMG_CUDA(cudaMemsetAsync(dw, 0, sizeof(float) * (size_t)rows * cout, st));
    PMG_CUDA(cudaMemsetAsync(dbias, 0, sizeof(float) * (size_t)cout, st));
    if (cin == 1) {
        const int ty = (g.dout + kWgY - 1) / kWgY, tx = (g.dout + kPatchX - 1) / kPatchX;
        const long long tiles = (long long)batch * g.dout * ty * tx;
        const int ps__ = prof_begin("k_conv1_wgrad", st);
        k_conv1_wgrad<<<dim3((unsigned)std::min<long long>(tiles, 152 * 8), cout / 16), 128, 0, st>>>(
            (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)dz, dw, dbias, di, g.dout, cout, ty, tx, (int)tiles);
        prof_end(ps__, 2.0 * np * cout * 27.0, st);
        PMG_CHECK_LAUNCH();
    } else {
        OpWgrad op;
        op.g = g;
        op.x = (const __nv_bfloat16 *)x;
        op.dz = (const __nv_bfloat16 *)dz;
        op.dw = dw;
        op.vec = !(reinterpret_cast<uintptr_t>(dw) & 15);
        op.kchunks_total = (int)((np + kBK - 1) / kBK);
        op.lgc = log2_of(cin);
        op.qo = fastdiv_of((unsigned)g.dout);
        const int mt = (int)((rows + kBM - 1) / kBM);
        // split K over about three CTAs per SM, but not below eight chunks
        // each: every split adds its whole tile with atomics
        const int ksplit = std::max(1, std::min(3 * 152 / mt, op.kchunks_total / 8));
        PMG_TRY((launch_tiles<OpWgrad, 64>(op, mt, ksplit, err, st, "k_umma_conv_wgrad", 2.0 * np * cout * 27.0 * cin)));
    }
    {
        const int ps__ = prof_begin("k_unpack_dw", st);
        k_unpack_dw<<<64, 256, 0, st>>>(dw, cin, cout, grad);
        prof_end(ps__, 0.0, st);
    }
    if (cin > 1) {
        const int ps__ = prof_begin("k_bias_grad", st);
        k_bias_grad<<<grid_for(np * (cout / 8), 256, 152LL * 4), 256, 0, st>>>((const __nv_bfloat16 *)dz, np, cout, dbias);
        prof_end(ps__, 0.0, st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

extern "C" int pmg_cnn_check(int32_t *err, void *stream) { return cnn_err_check(err, as_stream(stream)); }

extern "C" int pmg_cnn_head(const void *y4, const float *params, int32_t batch, const float *target, float *pred,
                            float *loss, float *grads, void *dy4, void *stream)
{
    if (!y4 || !params || !pred || batch <= 0 || (target && (!loss || !grads || !dy4))) {
        set_error("pmg_cnn_head: bad argument");
        return PMG_EINVAL;
    }
    cudaStream_t st = as_stream(stream);
    const float *w5 = params, *b5 = w5 + kHead * kHead, *w6 = b5 + kHead, *b6 = w6 + kHead * kHead;
    float *gw5 = grads, *gb5 = grads ? gw5 + kHead * kHead : nullptr, *gw6 = grads ? gb5 + kHead : nullptr,
          *gb6 = grads ? gw6 + kHead * kHead : nullptr;
    const int ps__ = prof_begin("k_head", st);
    k_head<<<batch, kHead, 0, st>>>((const __nv_bfloat16 *)y4, w5, b5, w6, b6, target, pred, loss, gw5, gb5, gw6,
                                    gb6, (__nv_bfloat16 *)dy4, 1.0f / (float)batch);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

extern "C" int pmg_cnn_adam(float *w, const float *g, float *m, float *v, int64_t n, double lr, double b1,
                            double b2, double eps, int64_t step, double weight_decay, void *stream)
{
    if (!w || !g || !m || !v || n <= 0 || step <= 0) {
        set_error("pmg_cnn_adam: bad argument");
        return PMG_EINVAL;
    }
    cudaStream_t st = as_stream(stream);
    const float c1 = (float)(1.0 - std::pow(b1, (double)step)), c2 = (float)(1.0 - std::pow(b2, (double)step));
    const int ps__ = prof_begin("k_adam", st);
    k_adam<<<152, 256, 0, st>>>(w, g, m, v, n, (float)lr, (float)b1, (float)b2, (float)eps, c1, c2,
                                (float)weight_decay);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

extern "C" int pmg_cnn_downsample(const float *dist, const int64_t shape[3], const int64_t box[6], double scale,
                                  void *out, void *stream)
{
    if (!dist || !shape || !box || !out || !(scale > 0.0)) {
        set_error("pmg_cnn_downsample: bad argument");
        return PMG_EINVAL;
    }
    const int l0 = (int)(box[1] - box[0]), l1 = (int)(box[3] - box[2]), l2 = (int)(box[5] - box[4]);
    if (l0 < 64 || l1 < 64 || l2 < 64 || box[0] < 0 || box[2] < 0 || box[4] < 0 || box[1] > shape[0] ||
        box[3] > shape[1] || box[5] > shape[2]) {
        set_error("pmg_cnn_downsample: box must lie in the volume and span at least 64 voxels per axis");
        return PMG_EINVAL;
    }
    cudaStream_t st = as_stream(stream);
    const int ps__ = prof_begin("k_downsample", st);
    k_downsample<<<64 * 64 * 64 / 256, 256, 0, st>>>(dist, shape[1], shape[2], (int)box[0], (int)box[2],
                                                     (int)box[4], l0, l1, l2, (float)(1.0 / scale),
                                                     (__nv_bfloat16 *)out);
    prof_end(ps__, (double)l0 * l1 * l2 * 4, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}
