// Capped integer morphology for isotropic power-of-two voxels (sm_103a).
//
// With a voxel size res = 2^k on every axis the reference's float32 squared
// distances are exact integer multiples of res^2 (src/pmmoto/filters/distance/
// _distance.hpp:135-272 performs only exact float operations on them, see
// edt_exact.cu), so the reference's test "sqrt(d2) <= r" (morphological_
// operators.py:103-228) is "E <= T" for the integer squared distance E and one
// integer bound T (morph_threshold).  Only values up to T matter, which gives
// a different, cheaper pipeline with the same result:
//
//   pass A (rows, the contiguous axis): E_A = min(d^2, T + 1), d the distance
//     to the nearest zero of the row -- one warp per row, ballots per chunk of
//     32 voxels, uint16 output;
//   pass B (axis 1, strided): E_B = min(E_A envelope, T + 1) -- one thread
//     per line, lanes on adjacent lines (coalesced), lower envelope of the
//     parabolas with E_A <= T, each output written a fixed W = floor(sqrt T)
//     positions behind the input (no later parabola can lower a value to <= T
//     after that), so all lanes store the same position; live parabolas lie
//     in [i - 2W, i] and fit a 64-entry ring when T <= 1023;
//   pass C (axis 0, strided): a height E_B <= T covers |x - v| <= floor(sqrt(
//     T - E_B)); x is within iff some interval covers it -- one thread per
//     line, a 64-bit window of pending positions, the result fused with the
//     unpadding and the wall rule.
//
// The exact squared EDT is separable in any axis order, so doing the linear
// pass on the contiguous axis leaves both envelope passes on strided axes,
// where a warp reads and writes 32 adjacent voxels at a time.  The reference's
// linear pass restarts at changes between nonzero values (multi-label
// images), which depends on the axis: this pipeline serves binary images only.
#include <type_traits>

#include "edt_internal.cuh"

namespace pmg {

struct CapGeo {
    int X0, X1, X2;       // extended shape
    int j0, nj, k0, nk;   // unextended ranges of axes 1 and 2
    int P2, PO;           // row pitch of the heights: X2 made even; of k_cap_mid's output
    // the voxel pairs that cover [k0, k0 + nk)
    __host__ __device__ int kp0() const { return k0 >> 1; }
    __host__ __device__ int np() const { return ((k0 + nk + 1) >> 1) - (k0 >> 1); }
};

// ---- x range of the seeds -------------------------------------------------------
// An optional block-plane range of the seeds (kRangeBig encoding, device
// memory): planes outside [hlo, hhi] hold no seed, so the row and envelope
// passes skip them, and the last pass produces only the outputs within W of
// the seeds, [olo, ohi] widened to whole 2x2x2 blocks.
struct SeedRange {
    int hlo, hhi, olo, ohi; // hlo > hhi: no seeds
    __device__ __forceinline__ void load(const int *xr, int n, int W)
    {
        const int a = xr[0], b = xr[1];
        if (a == 0) {
            hlo = olo = 2;
            hhi = ohi = -1;
            return;
        }
        hlo = 2 * (kRangeBig - b);
        hhi = min(2 * (a - 1) + 1, n - 1);
        olo = max(0, hlo - W) & ~1;
        ohi = min(n - 1, (hhi + W) | 1);
    }
};

// ---- pass A: rows -------------------------------------------------------------
// The seeds of a dilation are the nonzero voxels of the extended image off the
// wall planes, those of an erosion its zeros and the wall planes.  Rows come
// from the image's nonzero voxels as bits (in memory order; periodic axes read
// the own region modulo its length), or (dilations without periodic axes) from
// row words (b1, nt2: block rows and pieces of a row).
struct RowSrc {
    ExtGeo G;
    int dilate;
    const unsigned *bits;
    long long last; // last word of bits
    const unsigned *rows;
    int b1, nt2;
    FastDiv q1; // division by the extended rows of a plane
    FastDiv qp; // and by the words of a row of k_seed_bits
};

// minimum of both 16-bit halves
__device__ __forceinline__ uint32_t pair_min(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// bits 0-15 of v at the even positions
__device__ __forceinline__ unsigned spread16(unsigned v)
{
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    return (v | (v << 1)) & 0x55555555u;
}

// bits of the nonzero bytes of v
__device__ __forceinline__ unsigned nonzero4(unsigned v)
{
    const unsigned m = (((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) >> 7 & 0x01010101u;
    return (m * 0x204081u) >> 21 & 0xfu;
}

// Nonzero voxels of an image as bits in memory order; *nonbinary is set when a
// voxel above 1 is met (null: not asked).  A lane takes 16 bytes; bound by the
// image read.
__global__ void __launch_bounds__(256) k_image_bits(const uint8_t *__restrict__ img, unsigned *__restrict__ bits,
                                                    long long n, int *nonbinary)
{
    const int lane = threadIdx.x & 31;
    const bool aligned = !((uintptr_t)img & 15);
    unsigned above = 0;
    for (long long base = (blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31)) * 16; base < n;
         base += (long long)gridDim.x * blockDim.x * 16) {
        const long long at = base + 16 * lane;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (aligned && at + 16 <= n) {
            v = *reinterpret_cast<const uint4 *>(img + at);
        } else {
            unsigned w[4] = {0u, 0u, 0u, 0u};
            for (int e = 0; e < 16 && at + e < n; e++)
                w[e >> 2] |= (unsigned)img[at + e] << (8 * (e & 3));
            v = make_uint4(w[0], w[1], w[2], w[3]);
        }
        above |= (v.x | v.y | v.z | v.w) & 0xfefefefeu;
        unsigned w = nonzero4(v.x) | nonzero4(v.y) << 4 | nonzero4(v.z) << 8 | nonzero4(v.w) << 12;
        w |= __shfl_down_sync(0xffffffffu, w, 1) << 16;
        if (!(lane & 1) && at < n)
            bits[at >> 5] = w;
    }
    if (nonbinary && __any_sync(0xffffffffu, above) && lane == 0)
        *nonbinary = 1;
}

// Word c of the seeds of row r of the extended volume.
template <bool WORDS>
__device__ __forceinline__ unsigned seed_word(const RowSrc &rs, int r, int c, int X1, int X2)
{
    const int i = (int)fdiv((unsigned)r, rs.q1), j = r - i * X1;
    const ExtAxis &a2 = rs.G.ax[2];
    bool wrow = false;
    const int s0 = (int)src_index(rs.G.ax[0], i, wrow), s1 = (int)src_index(rs.G.ax[1], j, wrow);
    unsigned w = 0; // a wall row: no voxel
    if (!wrow) {
        if constexpr (WORDS) {
            // 64 voxels per piece: even positions in one word, odd ones in the next
            const uint2 eo = *reinterpret_cast<const uint2 *>(
                rs.rows + ((long long)((i >> 1) * rs.b1 + (j >> 1)) * rs.nt2 + (c >> 1)) * 8 + ((i & 1) * 2 + (j & 1)) * 2);
            const int sh = (c & 1) * 16;
            w = spread16((eo.x >> sh) & 0xffffu) | (spread16((eo.y >> sh) & 0xffffu) << 1);
        } else {
            const long long row = ((long long)s0 * rs.G.ax[1].S + s1) * a2.S;
            // bits from position p of the row (past its end: the next rows')
            auto bits_at = [&](int p) {
                const long long b = row + p;
                return __funnelshift_r(rs.bits[b >> 5], rs.bits[min((b >> 5) + 1, rs.last)], (unsigned)b & 31u);
            };
            if (!a2.periodic) {
                w = bits_at(32 * c);
            } else {
                int q = 32 * c - (a2.own_lo + a2.ext_lo);
                if (q < -a2.own_len || q >= a2.own_len)
                    q %= a2.own_len;
                q += q < 0 ? a2.own_len : 0;
                for (int f = 0; f < 32;) {
                    const int take = min(32 - f, a2.own_len - q);
                    w |= (bits_at(a2.own_lo + q) & (0xffffffffu >> (32 - take))) << f;
                    f += take;
                    q = 0;
                }
            }
        }
        if (!a2.periodic) {
            // the wall planes at the row's ends
            if (a2.wall_lo && c == 0)
                w &= ~1u;
            if (a2.wall_hi && c == (X2 - 1) >> 5)
                w &= ~(1u << ((X2 - 1) & 31));
        }
    }
    // seeds: the voxels, or (erosion) the others
    const unsigned in = X2 - 32 * c >= 32 ? 0xffffffffu : (1u << (X2 - 32 * c)) - 1u;
    return (rs.dilate ? w : ~w) & in;
}

// Squared distances, at most big, of two adjacent positions (the first at bit sh
// of wc, sh even) to the nearest set bits of their row's words wp, wc, wn: bit
// 31 - t of l holds the positions x - t and x + t.
__device__ __forceinline__ uint32_t pair_heights(uint32_t wp, uint32_t wc, uint32_t wn, int sh, uint32_t bigp)
{
    const uint32_t l0 = __funnelshift_l(wp, wc, 31 - sh) | __brev(__funnelshift_r(wc, wn, sh)),
                   l1 = __funnelshift_l(wp, wc, 30 - sh) | __brev(__funnelshift_r(wc, wn, sh + 1));
    const uint32_t d0 = __clz(l0), d1 = __clz(l1); // 32: none near, above every W
    return pair_min(d0 * d0 + d1 * d1 * 65536u, bigp);
}

// The seeds of the extended volume as bits: nw words per row between a zero word
// before and two behind (pitch nw + 3).  One thread per word.
template <bool WORDS>
__global__ void __launch_bounds__(256) k_seed_bits(RowSrc rs, unsigned *__restrict__ eb, int rows, int X2, int W,
                                                   const unsigned long long *__restrict__ gate,
                                                   const int *__restrict__ xr)
{
    if (gate && *gate == 0)
        return;
    const int X1 = (int)rs.G.ax[1].X, nw = (X2 + 31) >> 5, pitch = nw + 3;
    SeedRange sr{0, 0x7fffffff, 0, 0};
    if (xr)
        sr.load(xr, rows / X1, W);
    const int r0 = xr ? max(sr.hlo, 0) * X1 : 0, r1 = xr ? (int)min((long long)rows, (long long)(sr.hhi + 1) * X1) : rows;
    // (words of a volume: below 2^32)
    const long long n = (long long)max(r1 - r0, 0) * pitch;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int rr = (int)fdiv((unsigned)q, rs.qp), c = (int)((unsigned)q - (unsigned)rr * pitch) - 1, r = r0 + rr;
        eb[(long long)r * pitch + c + 1] = c >= 0 && c < nw ? seed_word<WORDS>(rs, r, c, X1, X2) : 0u;
    }
}

// Only distances d <= W = floor(sqrt T) <= 31 give values below T + 1, so a
// voxel needs the seeds within 31 positions on either side: the row's seed words
// are gathered in shared memory, with an empty word on either side, then every
// lane finds the nearest seeds of two adjacent voxels in the three words around
// them and stores both at once (rows of even pitch; the column that an odd row
// gains holds some height, read by no one).  For the wide probes only: the
// others' next pass takes the heights from the words itself.
template <bool WORDS>
__global__ void __launch_bounds__(256) k_cap_rows(RowSrc rs, uint16_t *__restrict__ KA, int rows, int X2, int T,
                                                  int W, const unsigned long long *__restrict__ gate,
                                                  const int *__restrict__ xr, unsigned long long *units)
{
    if (gate && *gate == 0)
        return; // empty seed set: the last pass writes the result alone
    const int X1 = (int)rs.G.ax[1].X;
    SeedRange sr{0, 0x7fffffff, 0, 0};
    if (xr)
        sr.load(xr, rows / X1, W);
    extern __shared__ uint32_t s_words[];
    const int lane = threadIdx.x & 31, nw = (X2 + 31) >> 5;
    uint32_t *zw = s_words + (threadIdx.x >> 5) * (nw + 3) + 1; // zw[-1], zw[nw] and zw[nw + 1] stay 0
    if (lane == 0) {
        zw[-1] = 0u;
        zw[nw] = 0u;
        zw[nw + 1] = 0u;
    }
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int P2 = (X2 + 1) & ~1;
    const uint32_t bigp = (uint32_t)(T + 1) * 0x10001u;
    // with a seed range, only the rows of its planes
    const int r0 = xr ? max(sr.hlo, 0) * X1 : 0;
    const int r1 = xr ? (int)min((long long)rows, (long long)(sr.hhi + 1) * X1) : rows;
    if (units && blockIdx.x == 0 && threadIdx.x == 0 && r1 > r0)
        atomicAdd(units, (unsigned long long)((long long)(r1 - r0) * X2));
    for (int r = r0 + warp; r < r1; r += nwarps) {
        for (int c = lane; c < nw; c += 32)
            zw[c] = seed_word<WORDS>(rs, r, c, X1, X2);
        __syncwarp();
        uint16_t *dst = KA + (long long)r * P2;
        // lane l on voxels 64 c + 2 l and the next one: word 2 c + l / 16
        const int hw = lane >> 4, sh = (2 * lane) & 31;
        for (int c = 0; 64 * c < X2; c++) {
            const int x = 64 * c + 2 * lane;
            const uint32_t v = pair_heights(zw[2 * c + hw - 1], zw[2 * c + hw], zw[2 * c + hw + 1], sh, bigp);
            if (x < X2)
                *reinterpret_cast<uint32_t *>(dst + x) = v;
        }
        __syncwarp();
    }
}

// The row pass: heights to KA, or (eb) the seeds' words there.  bits: scratch of a
// word per 32 voxels of the image; *nonbinary (erosions) is read back
// from flag.
static int launch_cap_rows(const uint8_t *img, const ExtGeo &EG, int dilate, const unsigned *seeds, unsigned *bits,
                           uint16_t *KA, bool eb, const CapGeo &G, int T, int W, int *flag, int *nonbinary,
                           cudaStream_t st, const unsigned long long *gate, const int *xr)
{
    const long long n = EG.ax[0].S * EG.ax[1].S * EG.ax[2].S;
    RowSrc rs{EG, dilate, bits, (n - 1) >> 5, seeds, (G.X1 + 1) / 2, ((G.X2 + 1) / 2 + 31) / 32,
              fastdiv_of((unsigned)G.X1), fastdiv_of((unsigned)((G.X2 + 31) / 32 + 3))};
    const int block = 256, rows = G.X0 * G.X1;
    if (flag)
        PMG_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
    if (!seeds) {
        const int ps__ = prof_begin("k_image_bits", st);
        k_image_bits<<<grid_for((n + 15) / 16, block, 152LL * 32), block, 0, st>>>(img, bits, n, flag);
        prof_end(ps__, (double)n * 1.125, st);
        PMG_CHECK_LAUNCH();
    }
    if (eb) {
        const int pitch = (G.X2 + 31) / 32 + 3;
        const unsigned grid = grid_for((long long)rows * pitch, block, 152LL * 32);
        const int ps__ = prof_begin("k_seed_bits", st);
        if (seeds)
            k_seed_bits<true><<<grid, block, 0, st>>>(rs, (unsigned *)KA, rows, G.X2, W, gate, xr);
        else
            k_seed_bits<false><<<grid, block, 0, st>>>(rs, (unsigned *)KA, rows, G.X2, W, gate, xr);
        prof_end(ps__, (double)rows * pitch * 8, st);
    } else {
        const size_t smem = (size_t)(block / 32) * ((G.X2 + 31) / 32 + 3) * sizeof(uint32_t);
        const unsigned grid = grid_for((long long)rows * 32, block, 152LL * 16);
        const int ps__ = prof_begin("k_cap_rows", st);
        if (seeds)
            k_cap_rows<true><<<grid, block, smem, st>>>(rs, KA, rows, G.X2, T, W, gate, xr, prof_units(kUnitsCapRows));
        else
            k_cap_rows<false><<<grid, block, smem, st>>>(rs, KA, rows, G.X2, T, W, gate, xr, prof_units(kUnitsCapRows));
        // 1/8 B read + 2 B written per voxel
        prof_end_units(ps__, kUnitsCapRows, 2.125, st);
    }
    PMG_CHECK_LAUNCH();
    if (flag) {
        PMG_CUDA(cudaMemcpyAsync(nonbinary, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
        PMG_CUDA(cudaStreamSynchronize(st));
    }
    return PMG_OK;
}

// ---- pass B: capped envelope along axis 1 --------------------------------------
// Ring entries pack a height (<= T <= 1023) and a vertex (< 2048): K << 11 | v.
__device__ __forceinline__ int cap_val(int ent, int x)
{
    const int d = x - (ent & 2047);
    return (ent >> 11) + d * d;
}

// Per-line state of the capped envelope; RING (a power of two) >= 2W + 2.
template <int RING>
struct CapLine {
    int *R; // ring slot s of this thread at R[s * 128]
    int bot, top, e;
    __device__ __forceinline__ int &at(int c) const { return R[(c & (RING - 1)) * 128]; }

    // consume height K at position i (K > T: absent), then return the value
    // at x = i - W (big when above T); x < 0 returns nothing meaningful
    __device__ __forceinline__ int step(int i, int K, int T, int W, int big)
    {
        if (K <= T) {
            while (top > bot) {
                const int t = at(top), u = at(top - 1);
                const int Kt = t >> 11, Vt = t & 2047, Ku = u >> 11, Vu = u & 2047;
                const int n1 = K - Kt + (i - Vt) * (i + Vt), d1 = 2 * (i - Vt);
                const int n2 = Kt - Ku + (Vt - Vu) * (Vt + Vu), d2 = 2 * (Vt - Vu);
                if (n1 * d2 > n2 * d1)
                    break;
                if (e == top)
                    e--;
                top--;
            }
            top++;
            at(top) = (K << 11) | i;
            if (top == bot)
                e = bot;
        }
        const int x = i - W;
        if (x < 0)
            return big;
        // parabolas with v + W < x exceed T at every later position
        while (bot <= top && (at(bot) & 2047) + W < x)
            bot++;
        if (e < bot)
            e = bot;
        if (top < bot)
            return big;
        int ce = at(e);
        while (e < top) {
            const int cn = at(e + 1);
            if (cap_val(cn, x) > cap_val(ce, x))
                break;
            ce = cn;
            e++;
        }
        const int Ev = cap_val(ce, x);
        return Ev <= T ? Ev : big;
    }
};

constexpr int kCapChunk = 8; // heights loaded ahead per line (memory-level parallelism)

// AX = 1: lines over (x0 in [0, X0), x2 in [k0, k0 + nk)) along axis 1;
// AX = 0: lines over (x1 in [j0, j0 + nj), x2 in [k0, k0 + nk)) along axis 0.
// One thread per line; each loop trip loads the next kCapChunk heights before
// it processes the current ones, so a thread keeps several loads in flight.
// Lines are cut into nseg segments: an output at x depends only on the
// heights within W of it, so a segment [a, b) is exact when its sweep starts
// at a - W (2W extra steps per segment buy nseg times the threads).
template <int AX, int RING>
__global__ void __launch_bounds__(128) k_cap_mid(const uint16_t *__restrict__ KA, uint16_t *__restrict__ KB,
                                                 CapGeo G, int T, int W, const unsigned long long *__restrict__ gate,
                                                 const int *__restrict__ xr, int nseg, unsigned long long *units)
{
    if (gate && *gate == 0)
        return;
    SeedRange sr{0, 0x7fffffff, 0, 0};
    if (xr)
        sr.load(xr, G.X0, W);
    __shared__ int ring[RING * 128];
    const long long nlines = (long long)(AX == 1 ? G.X0 : G.nj) * G.nk;
    const long long st = AX == 1 ? (long long)G.P2 : (long long)G.X1 * G.P2;
    const long long sto = AX == 1 ? (long long)G.PO : (long long)G.X1 * G.PO;
    const int n = AX == 1 ? G.X1 : G.X0;
    const int seglen = (n + nseg - 1) / nseg;
    const int big = T + 1;
    // with a seed range (axis-1 lines), only the lines of its planes
    const long long l0 = AX == 1 && xr ? (long long)max(sr.hlo, 0) * G.nk : 0;
    const long long l1 = AX == 1 && xr ? min(nlines, (long long)(sr.hhi + 1) * G.nk) : nlines;
    const long long span = l1 > l0 ? l1 - l0 : 0;
    if (units && blockIdx.x == 0 && threadIdx.x == 0 && span)
        atomicAdd(units, (unsigned long long)(span * n));
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < span * nseg;
         g += (long long)gridDim.x * blockDim.x) {
        const int seg = (int)(g / span);
        const long long li = l0 + (g - (long long)seg * span);
        const long long q = li / G.nk;
        const int a = seg * seglen, b = min(n, a + seglen);
        if (a >= b)
            continue;
        const int x2 = G.k0 + (int)(li - q * G.nk);
        const long long lrow = AX == 1 ? q * G.X1 : G.j0 + q;
        const uint16_t *in = KA + lrow * G.P2 + x2;
        uint16_t *out = KB + lrow * G.PO + x2;
        CapLine<RING> L{ring + threadIdx.x, 0, -1, 0};
        const int i_first = max(0, a - W), i_last = b - 1 + W; // steps; step i emits x = i - W
        int cur[kCapChunk];
        const uint16_t *pin = in + (long long)i_first * st; // next height to prefetch
#pragma unroll
        for (int u = 0; u < kCapChunk; u++) {
            cur[u] = i_first + u < n ? (int)*pin : big;
            pin += st;
        }
        uint16_t *po = out + (long long)a * sto; // output position x = i - W
        for (int i0 = i_first; i0 <= i_last; i0 += kCapChunk) {
            int nxt[kCapChunk];
#pragma unroll
            for (int u = 0; u < kCapChunk; u++) {
                nxt[u] = i0 + kCapChunk + u < n ? (int)*pin : big;
                pin += st;
            }
#pragma unroll
            for (int u = 0; u < kCapChunk; u++) {
                const int i = i0 + u;
                const int v = L.step(i, cur[u], T, W, big);
                const int x = i - W;
                if (x >= a && x < b) {
                    *po = (uint16_t)v;
                    po += sto;
                }
            }
#pragma unroll
            for (int u = 0; u < kCapChunk; u++)
                cur[u] = nxt[u];
        }
    }
}

// ---- pass B for small W: direct minima on line pairs ----------------------------
// E_B(y) = min over |d| <= W of E_A(y + d) + d^2: heights above T are stored
// as T + 1 and every term with |d| > W exceeds T, so the capped envelope is
// this minimum over 2W + 1 terms.  Two adjacent lines (x2 and x2 + 1) share a
// thread, packed in the halves of a 32-bit word, and each pair of terms costs
// two packed add-min instructions (values stay below 2^11: no carries between
// the halves).  The heights of a segment live in a register ring of
// R = 2W + 1 + pair_ahead(W) words whose slots are fixed at compile time: at
// step u of a group of R outputs starting at y0, slot s holds position
// y0 - W + s (s >= u) or y0 - W + s + R (s < u), so the term at y + d sits in
// slot (u + W + d) mod R, and the slot of y - W, dead after output y, takes
// position y + W + 1 + pair_ahead(W) (loaded that many steps before its use).
constexpr int kPairMaxW = 20;
// heights loaded ahead: fewer for the wide windows, whose rings hold more
__host__ __device__ constexpr int pair_ahead(int W) { return W <= 12 ? 8 : 4; }

// Along axis 0 (pairs over x1 in [j0, j0 + nj), x2 / 2 from kp0).
template <int W>
__global__ void __launch_bounds__(256) k_cap_mid_pair(const uint16_t *__restrict__ KA, uint16_t *__restrict__ KB,
                                                      CapGeo G, int T, int seglen, unsigned long long *units)
{
    constexpr int R = 2 * W + 1 + pair_ahead(W);
    const int np = G.np(), n = G.X0;
    const long long span = (long long)G.nj * np, st = (long long)G.X1 * (G.P2 >> 1);
    const int nseg = (n + seglen - 1) / seglen;
    if (units && blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(units, (unsigned long long)(span * 2 * n));
    const uint32_t bigp = (uint32_t)(T + 1) * 0x10001u;
    const uint32_t *in0 = (const uint32_t *)KA;
    uint32_t *out0 = (uint32_t *)KB;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < span * nseg;
         g += (long long)gridDim.x * blockDim.x) {
        const int seg = (int)(g / span);
        const long long li = g - (long long)seg * span, q = li / np;
        const long long base = (G.j0 + q) * (G.P2 >> 1) + G.kp0() + (li - q * np);
        const uint32_t *in = in0 + base;
        uint32_t *out = out0 + base;
        const int a = seg * seglen, b = min(n, a + seglen);
        uint32_t win[R];
#pragma unroll
        for (int s = 0; s < R; s++) {
            const int y = a - W + s;
            win[s] = y >= 0 && y < n ? __ldg(in + y * st) : bigp;
        }
        for (int y0 = a; y0 < b; y0 += R) {
#pragma unroll
            for (int u = 0; u < R; u++) {
                const int y = y0 + u;
                uint32_t m = win[(u + W) % R];
#pragma unroll
                for (int d = 1; d <= W; d++) {
                    const uint32_t dd = (uint32_t)(d * d) * 0x10001u;
                    m = __viaddmin_u16x2(win[(u + W - d) % R], dd, m);
                    m = __viaddmin_u16x2(win[(u + W + d) % R], dd, m);
                }
                if (y < b)
                    out[y * st] = m;
                const int yn = y + W + 1 + pair_ahead(W);
                win[u] = y < b && yn < n ? __ldg(in + yn * st) : bigp;
            }
        }
    }
}

// Passes A and B in one for small W: the heights of a position are taken from
// the three seed words around it (k_seed_bits) where the ring needs them, so
// neither written nor read.  The words of the next height are loaded a step
// ahead; a warp's 64 voxels share two to three words of a row.
// Bound by instruction issue.  As two passes (heights written, then read) this
// took 108 + 105 us a radius of the 512^3 drainage, and 55 + 23 us on 256 x 192 x
// 320 voxels.
template <int W>
__global__ void __launch_bounds__(256) k_cap_rows_mid(const unsigned *__restrict__ eb, uint16_t *__restrict__ KB,
                                                      CapGeo G, int T, const unsigned long long *__restrict__ gate,
                                                      const int *__restrict__ xr, int seglen,
                                                      unsigned long long *units)
{
    constexpr int R = 2 * W + 1;
    if (gate && *gate == 0)
        return;
    SeedRange sr{0, 0x7fffffff, 0, 0};
    if (xr)
        sr.load(xr, G.X0, W);
    const int np = G.np(), n = G.X1, pitch = ((G.X2 + 31) >> 5) + 3;
    const long long nlines = (long long)G.X0 * np, st = G.P2 >> 1;
    const int nseg = (n + seglen - 1) / seglen;
    const long long l0 = xr ? (long long)max(sr.hlo, 0) * np : 0;
    const long long l1 = xr ? min(nlines, (long long)(sr.hhi + 1) * np) : nlines;
    const long long span = l1 > l0 ? l1 - l0 : 0;
    if (units && blockIdx.x == 0 && threadIdx.x == 0 && span)
        atomicAdd(units, (unsigned long long)(span * 2 * n));
    const uint32_t bigp = (uint32_t)(T + 1) * 0x10001u;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < span * nseg;
         g += (long long)gridDim.x * blockDim.x) {
        const int seg = (int)(g / span);
        const long long li = l0 + (g - (long long)seg * span), q = li / np;
        const int kp = G.kp0() + (int)(li - q * np), x = 2 * kp, sh = x & 31;
        const unsigned *in = eb + q * n * pitch + (x >> 5);
        uint32_t *out = (uint32_t *)KB + q * n * st + kp;
        const int a = seg * seglen, b = min(n, a + seglen);
        uint32_t w[3];
        auto fetch = [&](int y) {
            const bool ok = y >= 0 && y < n;
            const unsigned *p = in + (long long)y * pitch;
#pragma unroll
            for (int c = 0; c < 3; c++)
                w[c] = ok ? __ldg(p + c) : 0u;
        };
        uint32_t win[R];
#pragma unroll
        for (int s = 0; s < R; s++) {
            fetch(a - W + s);
            win[s] = pair_heights(w[0], w[1], w[2], sh, bigp);
        }
        fetch(a + W + 1);
        for (int y0 = a; y0 < b; y0 += R) {
#pragma unroll
            for (int u = 0; u < R; u++) {
                const int y = y0 + u;
                uint32_t m = win[(u + W) % R];
#pragma unroll
                for (int d = 1; d <= W; d++) {
                    const uint32_t dd = (uint32_t)(d * d) * 0x10001u;
                    m = __viaddmin_u16x2(win[(u + W - d) % R], dd, m);
                    m = __viaddmin_u16x2(win[(u + W + d) % R], dd, m);
                }
                if (y < b)
                    out[y * st] = m;
                // the slot of y - W takes y + W + 1
                win[u] = pair_heights(w[0], w[1], w[2], sh, bigp);
                fetch(y < b ? y + W + 2 : n);
            }
        }
    }
}

// ---- pass C: intervals along axis 0, fused epilogue ----------------------------
__device__ __forceinline__ int isqrt_small(int m)
{
    int r = (int)__fsqrt_rn((float)m);
    if (r * r > m)
        r--;
    else if ((r + 1) * (r + 1) <= m)
        r++;
    return r;
}

// gate: a count of the seeds held in device memory (null: always seeds); when
// it is zero the dilation is empty and only zeros are written.
// Lines are cut into nseg segments of outputs, each swept from W positions
// before its first output (heights farther away cannot reach it).
__global__ void __launch_bounds__(128) k_cap_last(const uint16_t *__restrict__ KB, CapGeo G, int T, int W,
                                                  MorphEpi me, const unsigned long long *__restrict__ gate,
                                                  const int *__restrict__ xr, int *__restrict__ orange, int nseg,
                                                  unsigned long long *units)
{
    SeedRange sr{0, G.X0 - 1, 0, G.X0 - 1};
    if (xr)
        sr.load(xr, G.X0, W);
    if (gate && *gate == 0) {
        sr.olo = 2;
        sr.ohi = -1;
    }
    if (orange && blockIdx.x == 0 && threadIdx.x == 0) {
        orange[0] = sr.olo;
        orange[1] = sr.ohi;
    }
    if (xr && sr.olo > sr.ohi)
        return; // nothing within reach of a seed: the caller reads no output
    if (gate && *gate == 0) {
        const long long nl = (long long)me.o1 * me.o2, no = me.o0 * nl;
        for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < no;
             q += (long long)gridDim.x * blockDim.x)
            me.out[q] = 0;
        return;
    }
    // half-width of the interval of every height K <= T: floor(sqrt(T - K))
    __shared__ uint8_t s_w[kCapMaxT + 1];
    for (int q = threadIdx.x; q <= T; q += blockDim.x)
        s_w[q] = (uint8_t)isqrt_small(T - q);
    __syncthreads();
    const long long nlines = (long long)G.nj * G.nk;
    const long long st = (long long)G.X1 * G.P2;
    const int n = G.X0;
    // positions x of the line that lie in the unextended volume (and in the
    // output range of the seeds)
    const int xlo = max(max(0, me.e0), sr.olo), xhi = min(min(n, me.e0 + (int)me.o0), sr.ohi + 1);
    if (units && blockIdx.x == 0 && threadIdx.x == 0 && xhi > xlo)
        atomicAdd(units, (unsigned long long)(nlines * (xhi - xlo)));
    const int seglen = (n + nseg - 1) / nseg;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nlines * nseg;
         g += (long long)gridDim.x * blockDim.x) {
        const int seg = (int)(g / nlines);
        const long long li = g - (long long)seg * nlines;
        // this segment's outputs [ax, bx); heights exist on [sr.hlo, sr.hhi]
        // only, and the sweep starts W steps before the first output
        const int ax = max(xlo, seg * seglen), bx = min(xhi, (seg + 1) * seglen);
        if (ax >= bx)
            continue;
        const int istart = max(0, ax - W), iend = bx - 1 + W;
        const int x1 = G.j0 + (int)(li / G.nk);
        const int x2 = G.k0 + (int)(li - (li / G.nk) * G.nk);
        const uint16_t *in = KB + (long long)x1 * G.P2 + x2;
        const long long jo = x1 - me.e1, ko = x2 - me.e2;
        const bool wall_jk = (me.wall[2] && jo == 0) || (me.wall[3] && jo == me.o1 - 1) ||
                             (me.wall[4] && ko == 0) || (me.wall[5] && ko == me.o2 - 1);
        const long long ost = me.o1 * me.o2;
        uint8_t *dst = me.out + jo * me.o2 + ko + (long long)(ax - me.e0) * ost; // output of x = ax
        // wall planes of axis 0 (unextended coordinates 0 and o0 - 1)
        const int xw0 = me.wall[0] ? me.e0 : -1, xw1 = me.wall[1] ? me.e0 + (int)me.o0 - 1 : -1;
        const uint8_t in_v = me.dilate ? 1 : 0, out_v = me.dilate ? 0 : 1;
        uint64_t pend = 0; // bit b: position i - b is covered
        int reach = -1;
        const int big = T + 1;
        const int hend = min(n, sr.hhi + 1); // heights are read on [hlo, hend)
        int cur[kCapChunk];
        const uint16_t *pin = in + (long long)istart * st;
#pragma unroll
        for (int u = 0; u < kCapChunk; u++) {
            const int i = istart + u;
            cur[u] = i >= sr.hlo && i < hend ? (int)*pin : big;
            pin += st;
        }
        for (int i0 = istart; i0 <= iend; i0 += kCapChunk) {
            int nxt[kCapChunk];
#pragma unroll
            for (int u = 0; u < kCapChunk; u++) {
                const int i = i0 + kCapChunk + u;
                nxt[u] = i >= sr.hlo && i < hend ? (int)*pin : big;
                pin += st;
            }
#pragma unroll
            for (int u = 0; u < kCapChunk; u++) {
                const int i = i0 + u;
                pend <<= 1;
                const int K = cur[u]; // big past the end of the line
                if (K <= T) {
                    const int w = s_w[K];
                    pend |= (2ull << w) - 1ull;
                    reach = max(reach, i + w);
                }
                if (reach >= i && i < n)
                    pend |= 1ull;
                const int x = i - W;
                if (x < ax || x >= bx)
                    continue;
                uint8_t v = ((pend >> W) & 1ull) ? in_v : out_v;
                if (wall_jk || x == xw0 || x == xw1)
                    v = 0;
                *dst = v;
                dst += ost;
            }
#pragma unroll
            for (int u = 0; u < kCapChunk; u++)
                cur[u] = nxt[u];
        }
    }
}

// Pass C for small W on line pairs (pairs over (x1 in [j0, j0 + nj), x2 / 2)
// along axis 0): x is within iff min over |d| <= W of E_B(x + d) + d^2 <= T,
// the same test as the intervals of k_cap_last, then the same epilogue; the
// two outputs of a pair are stored as one 16-bit word where o2 and x2 - e2 are
// even, else byte by byte.
// ROWS: as row words instead (no extension) -- a warp holds 64 voxels of one
// row, whose even and odd ones are two ballots, 1 bit written per voxel; each
// row's pairs are padded to whole warps.
template <int W, bool ROWS>
__global__ void __launch_bounds__(256) k_cap_last_pair(const uint16_t *__restrict__ KB, CapGeo G, int T, MorphEpi me,
                                                       const unsigned long long *__restrict__ gate,
                                                       const int *__restrict__ xr, int *__restrict__ orange,
                                                       int seglen, unsigned *__restrict__ rows_out,
                                                       unsigned long long *units)
{
    constexpr int R = 2 * W + 1 + pair_ahead(W);
    SeedRange sr{0, G.X0 - 1, 0, G.X0 - 1};
    if (xr)
        sr.load(xr, G.X0, W);
    if (gate && *gate == 0) {
        sr.olo = 2;
        sr.ohi = -1;
    }
    if (orange && blockIdx.x == 0 && threadIdx.x == 0) {
        orange[0] = sr.olo;
        orange[1] = sr.ohi;
    }
    if (xr && sr.olo > sr.ohi)
        return; // nothing within reach of a seed: the caller reads no output
    if (gate && *gate == 0) {
        if constexpr (!ROWS) {
            const long long nl = (long long)me.o1 * me.o2, no = me.o0 * nl;
            for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < no;
                 q += (long long)gridDim.x * blockDim.x)
                me.out[q] = 0;
        }
        return;
    }
    const int np0 = G.np(), np = ROWS ? (np0 + 31) & ~31 : np0;
    const long long nlines = (long long)G.nj * np;
    const long long st = (long long)G.X1 * (G.P2 >> 1);
    const int n = G.X0;
    const int xlo = max(max(0, me.e0), sr.olo), xhi = min(min(n, me.e0 + (int)me.o0), sr.ohi + 1);
    if (xhi <= xlo)
        return;
    if (units && blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(units, (unsigned long long)(nlines * 2 * (xhi - xlo)));
    const int nseg = (xhi - xlo + seglen - 1) / seglen;
    const int hlo = sr.hlo, hend = min(n, sr.hhi + 1); // heights are read on [hlo, hend)
    // (a minimum is at most T + 1, its own term, and T + 1 only out of reach)
    const uint32_t bigp = (uint32_t)(T + 1) * 0x10001u, lim = (uint32_t)(T + 1) << 16;
    const long long ost = me.o1 * me.o2;
    const int xw0 = me.wall[0] ? me.e0 : -1, xw1 = me.wall[1] ? me.e0 + (int)me.o0 - 1 : -1;
    const uint32_t *in0 = (const uint32_t *)KB;
    const bool odd = (me.o2 | me.e2) & 1; // pairs do not start on even output bytes
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nlines * nseg;
         g += (long long)gridDim.x * blockDim.x) {
        const int seg = (int)(g / nlines);
        const long long li = g - (long long)seg * nlines;
        const int a = xlo + seg * seglen, b = min(xhi, a + seglen);
        const long long q = li / np;
        const int x1 = G.j0 + (int)q;
        const int kp = (int)(li - q * np);
        const bool live = !ROWS || kp < np0;
        const int x2 = 2 * (G.kp0() + kp);
        // (the padding lanes read the row's last pair and write no bit)
        const uint32_t *in = in0 + (G.j0 + q) * (G.P2 >> 1) + G.kp0() + (ROWS ? min(kp, np0 - 1) : kp);
        const long long jo = x1 - me.e1, ko = x2 - me.e2;
        const bool wall_j = (me.wall[2] && jo == 0) || (me.wall[3] && jo == me.o1 - 1);
        // bytes of the pair inside the output and off the wall lines
        const bool in0k = live && ko >= 0, in1k = live && ko + 1 < me.o2;
        auto wall_k = [&](long long k) { return (me.wall[4] && k == 0) || (me.wall[5] && k == me.o2 - 1); };
        const uint32_t keep = (!in0k || wall_j || wall_k(ko) ? 0u : 0x00ffu) |
                              (!in1k || wall_j || wall_k(ko + 1) ? 0u : 0xff00u);
        uint8_t *dst = me.out + jo * me.o2 + ko + (long long)(a - me.e0) * ost;
        uint32_t win[R];
#pragma unroll
        for (int s = 0; s < R; s++) {
            const int y = a - W + s;
            win[s] = y >= hlo && y < hend ? __ldg(in + y * st) : bigp;
        }
        // this warp's two words of a plane: z = 0 and 1 of its 32 blocks
        unsigned *rw = nullptr;
        if constexpr (ROWS)
            rw = rows_out + ((long long)(x1 >> 1) * (np >> 5) + (kp >> 5)) * 8 + (x1 & 1) * 2 + (threadIdx.x & 1);
        const int plane = ((G.nj + 1) >> 1) * (np >> 5) * 8;
        const unsigned keep0 = ROWS ? __ballot_sync(0xffffffffu, keep & 1u) : 0u,
                       keep1 = ROWS ? __ballot_sync(0xffffffffu, keep & 0x100u) : 0u;
        for (int y0 = a; y0 < b; y0 += R) {
#pragma unroll
            for (int u = 0; u < R; u++) {
                const int y = y0 + u;
                uint32_t m = win[(u + W) % R];
#pragma unroll
                for (int d = 1; d <= W; d++) {
                    const uint32_t dd = (uint32_t)(d * d) * 0x10001u;
                    m = __viaddmin_u16x2(win[(u + W - d) % R], dd, m);
                    m = __viaddmin_u16x2(win[(u + W + d) % R], dd, m);
                }
                if (y < b) {
                    const bool hit0 = (m << 16) < lim, hit1 = m < lim; // within reach
                    if constexpr (ROWS) {
                        const unsigned w0 = __ballot_sync(0xffffffffu, hit0) & keep0,
                                       w1 = __ballot_sync(0xffffffffu, hit1) & keep1;
                        if ((threadIdx.x & 31) < 2)
                            rw[(long long)(y >> 1) * plane + (y & 1) * 4] = threadIdx.x & 1 ? w1 : w0;
                    } else {
                        uint32_t v = (hit0 ? 1u : 0u) | (hit1 ? 0x100u : 0u);
                        if (!me.dilate)
                            v ^= 0x101u;
                        v &= keep;
                        if (y == xw0 || y == xw1)
                            v = 0u;
                        if (!odd) {
                            *reinterpret_cast<uint16_t *>(dst) = (uint16_t)v;
                        } else {
                            if (in0k)
                                dst[0] = (uint8_t)v;
                            if (in1k)
                                dst[1] = (uint8_t)(v >> 8);
                        }
                        dst += ost;
                    }
                }
                const int yn = y + W + 1 + pair_ahead(W);
                win[u] = y < b && yn >= hlo && yn < hend ? __ldg(in + yn * st) : bigp;
            }
        }
        if constexpr (ROWS) {
            // the wall planes, by the threads that wrote them
            if ((threadIdx.x & 31) < 2) {
                if (xw0 >= a && xw0 < b)
                    rw[(long long)(xw0 >> 1) * plane + (xw0 & 1) * 4] = 0u;
                if (xw1 >= a && xw1 < b)
                    rw[(long long)(xw1 >> 1) * plane + (xw1 & 1) * 4] = 0u;
            }
        }
    }
}

// Segment length of the pair kernels on `lines` lines of n: whole groups of the
// register ring of R, four per segment, as each starts with a ring to fill, and
// fewer (two at least) where that leaves less than about six warps per scheduler
// (200^3 voxels: 29 + 26 us for the two passes with four, 24 + 21 us with two).
static int pair_seglen(int R, int n, long long lines)
{
    int g = 4;
    while (g > 2 && lines * ((n + g * R - 1) / (g * R)) < 152LL * 768)
        g--;
    return g * R;
}

// Calls f with std::integral_constant<int, w> for 0 <= w <= kPairMaxW.
template <int W, class F>
static void with_w(int w, F &&f)
{
    if constexpr (W < kPairMaxW) {
        if (w > W) {
            with_w<W + 1>(w, f);
            return;
        }
    }
    f(std::integral_constant<int, W>{});
}

static void launch_mid_pair(const uint16_t *in, uint16_t *out, const CapGeo &G, int T, int W, cudaStream_t st,
                            unsigned long long *units)
{
    with_w<0>(W, [&](auto c) {
        constexpr int w = decltype(c)::value;
        const int seglen = pair_seglen(2 * w + 1 + pair_ahead(w), G.X0, (long long)G.nj * G.np());
        const long long work = (long long)G.nj * G.np() * ((G.X0 + seglen - 1) / seglen);
        k_cap_mid_pair<w><<<grid_for(work, 256, 1LL << 30), 256, 0, st>>>(in, out, G, T, seglen, units);
    });
}

// The two passes in one (words: the seeds' words in KA) where the window fits the
// registers and the words fit the heights' scratch.
static bool rows_mid_ok(const CapGeo &G, int W) { return W <= kPairMaxW && G.X2 >= 4; }

static int launch_rows_mid(const uint16_t *KA, uint16_t *KB, const CapGeo &G, int T, int W, cudaStream_t st,
                           const unsigned long long *gate, const int *xr)
{
    const int ps__ = prof_begin("k_cap_rows_mid", st);
    with_w<0>(W, [&](auto c) {
        constexpr int w = decltype(c)::value;
        const int seglen = pair_seglen(2 * w + 1, G.X1, (long long)G.X0 * G.np());
        const long long work = (long long)G.X0 * G.np() * ((G.X1 + seglen - 1) / seglen);
        k_cap_rows_mid<w><<<grid_for(work, 256, 1LL << 30), 256, 0, st>>>((const unsigned *)KA, KB, G, T, gate, xr, seglen,
                                                                         prof_units(kUnitsCapMid));
    });
    prof_end_units(ps__, kUnitsCapMid, 2.125, st); // 1/8 B read + 2 B written per voxel
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

template <int W>
static void launch_last_pair_w(const uint16_t *KB, const CapGeo &G, int T, const MorphEpi &me, cudaStream_t st,
                               const unsigned long long *gate, const int *xr, int *orange, unsigned *rows_out,
                               unsigned long long *units)
{
    const long long np = rows_out ? (G.np() + 31) & ~31 : G.np();
    const int seglen = pair_seglen(2 * W + 1 + pair_ahead(W), G.X0, G.nj * np);
    const long long work = G.nj * np * ((G.X0 + seglen - 1) / seglen);
    const unsigned grid = grid_for(work, 256, 1LL << 30);
    if (rows_out)
        k_cap_last_pair<W, true><<<grid, 256, 0, st>>>(KB, G, T, me, gate, xr, orange, seglen, rows_out, units);
    else
        k_cap_last_pair<W, false><<<grid, 256, 0, st>>>(KB, G, T, me, gate, xr, orange, seglen, nullptr, units);
}

static void launch_last_pair(const uint16_t *KB, const CapGeo &G, int T, int W, const MorphEpi &me, cudaStream_t st,
                             const unsigned long long *gate, const int *xr, int *orange, unsigned *rows_out,
                             unsigned long long *units)
{
    with_w<0>(W, [&](auto c) {
        launch_last_pair_w<decltype(c)::value>(KB, G, T, me, st, gate, xr, orange, rows_out, units);
    });
}

// Line pairs: windows that fit the registers, output rows of the same pitch.
static bool pair_ok(const CapGeo &G, int W) { return W <= kPairMaxW && G.PO == G.P2; }

// the ring holds the live parabolas, at most 2W + 2
template <int AX>
static int launch_cap_mid(const uint16_t *in, uint16_t *out, const CapGeo &G, int T, int W, long long lines,
                          cudaStream_t st, const unsigned long long *gate = nullptr, const int *xr = nullptr)
{
    // segments of at least 4 W + 32 positions, at most 4 per line
    const int n = AX == 1 ? G.X1 : G.X0;
    int nseg = n / (4 * W + 32);
    nseg = nseg < 1 ? 1 : nseg > 4 ? 4 : nseg;
    const unsigned grid = grid_for(lines * nseg, 128, 1LL << 30);
    // axis-1 passes count their voxels (k_cap_mid); the axis-0 pass of the
    // erosion EDT (k_cap_mid0) is booked from the host
    unsigned long long *units = AX == 1 ? prof_units(kUnitsCapMid) : nullptr;
    if constexpr (AX == 0) // (along axis 1: k_cap_rows_mid)
        if (pair_ok(G, W)) {
            launch_mid_pair(in, out, G, T, W, st, units);
            return PMG_OK;
        }
    if (2 * W + 2 <= 16)
        k_cap_mid<AX, 16><<<grid, 128, 0, st>>>(in, out, G, T, W, gate, xr, nseg, units);
    else if (2 * W + 2 <= 32)
        k_cap_mid<AX, 32><<<grid, 128, 0, st>>>(in, out, G, T, W, gate, xr, nseg, units);
    else
        k_cap_mid<AX, 64><<<grid, 128, 0, st>>>(in, out, G, T, W, gate, xr, nseg, units);
    return PMG_OK;
}

bool cap_path_ok(const float *res, const int64_t *X, int T)
{
    if (!(res[0] == res[1] && res[1] == res[2]) || T < 0 || T > kCapMaxT)
        return false;
    const pmg_axis_cfg plain = {0, 0, 0, 0, 1, 0, 0, 0};
    for (int d = 0; d < 3; d++)
        if (!exact_path_ok(res[d], plain, (int)X[d]))
            return false;
    return true;
}

bool cap_rows_out(const int64_t *X, int T, const MorphEpi &me)
{
    int W = 0;
    while ((W + 1) * (W + 1) <= T)
        W++;
    const bool plain = me.e0 == 0 && me.e1 == 0 && me.e2 == 0 && me.o0 == X[0] && me.o1 == X[1] && me.o2 == X[2];
    return plain && me.dilate && W <= kPairMaxW;
}

int morph_cap_run(const uint8_t *img, const ExtGeo &EG, uint16_t *KA, uint16_t *KB, const int64_t *X, int T,
                  const MorphEpi &me, cudaStream_t st, int *flag, int *nonbinary, const unsigned long long *gate,
                  const int *xr, int *orange, const unsigned *seeds, unsigned *rows_out)
{
    int W = 0;
    while ((W + 1) * (W + 1) <= T)
        W++;
    CapGeo G;
    G.X0 = (int)X[0];
    G.X1 = (int)X[1];
    G.X2 = (int)X[2];
    G.j0 = me.e1;
    G.nj = (int)me.o1;
    G.k0 = me.e2;
    G.nk = (int)me.o2;
    G.P2 = G.PO = (G.X2 + 1) & ~1;
    const bool fused = rows_mid_ok(G, W);
    PMG_TRY(launch_cap_rows(img, EG, me.dilate, seeds, (unsigned *)KB, KA, fused, G, T, W, flag, nonbinary, st, gate, xr));
    if (flag && *nonbinary)
        return PMG_OK;
    if (fused) {
        PMG_TRY(launch_rows_mid(KA, KB, G, T, W, st, gate, xr));
    } else {
        const long long lines = (long long)G.X0 * G.nk;
        const int ps__ = prof_begin("k_cap_mid", st);
        PMG_TRY(launch_cap_mid<1>(KA, KB, G, T, W, lines, st, gate, xr));
        prof_end_units(ps__, kUnitsCapMid, 4.0, st); // 2 B read + 2 B written per voxel
    }
    PMG_CHECK_LAUNCH();
    {
        const long long lines = (long long)G.nj * G.nk;
        const int ps__ = prof_begin("k_cap_last", st);
        // one segment per line: this pass is short per voxel, the extra sweep
        // of a cut costs more than the threads it adds
        const int nseg = 1;
        if (pair_ok(G, W))
            launch_last_pair(KB, G, T, W, me, st, gate, xr, orange, rows_out, prof_units(kUnitsCapLast));
        else
            k_cap_last<<<grid_for(lines * nseg, 128, 1LL << 30), 128, 0, st>>>(KB, G, T, W, me, gate, xr, orange,
                                                                               nseg, prof_units(kUnitsCapLast));
        prof_end_units(ps__, kUnitsCapLast, rows_out ? 2.125 : 3.0, st); // 2 B read + 1 B (1 bit) written per output
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// Capped squared EDT of a binary image (nothing is written when it is not):
// E = min(exact d^2
// in units of res^2, T + 1) as uint16, all three passes on the same volume.
int edt_cap_run(const uint8_t *img, const ExtGeo &EG, uint16_t *KA, uint16_t *KB, uint16_t *KC, const int64_t *X, int T,
                int *flag, int *nonbinary, cudaStream_t st)
{
    int W = 0;
    while ((W + 1) * (W + 1) <= T)
        W++;
    CapGeo G;
    G.X0 = (int)X[0];
    G.X1 = (int)X[1];
    G.X2 = (int)X[2];
    G.j0 = 0;
    G.nj = G.X1;
    G.k0 = 0;
    G.nk = G.X2;
    G.P2 = G.PO = (G.X2 + 1) & ~1;
    const long long vox = (long long)G.X0 * G.X1 * G.X2;
    const bool fused = rows_mid_ok(G, W);
    PMG_TRY(launch_cap_rows(img, EG, 0, nullptr, (unsigned *)KB, KA, fused, G, T, W, flag, nonbinary, st, nullptr,
                            nullptr));
    if (*nonbinary)
        return PMG_OK;
    if (fused) {
        PMG_TRY(launch_rows_mid(KA, KB, G, T, W, st, nullptr, nullptr));
    } else {
        const long long lines = (long long)G.X0 * G.nk;
        const int ps__ = prof_begin("k_cap_mid", st);
        PMG_TRY(launch_cap_mid<1>(KA, KB, G, T, W, lines, st));
        prof_end_units(ps__, kUnitsCapMid, 4.0, st);
    }
    PMG_CHECK_LAUNCH();
    {
        const long long lines = (long long)G.nj * G.nk;
        const int ps__ = prof_begin("k_cap_mid0", st);
        G.PO = G.X2; // the caller's volume
        PMG_TRY(launch_cap_mid<0>(KB, KC, G, T, W, lines, st));
        prof_end(ps__, (double)vox * 4, st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

} // namespace pmg
