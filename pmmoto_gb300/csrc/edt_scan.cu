// Envelope passes of any voxel size as an outward scan (sm_103a).
//
// The reference's lower envelope (squared_edt_1d_parabolic, _distance.hpp:
// 184-272) gives at every position x the float value a (x - v)^2 + f(v) of one
// parabola v, chosen by float intersections.  Each intersection s(r, q) is off
// by at most
//     2^-24 (4 |f_r - f_q| / (2 a (r - q)) + 3 (r + q) / 2),
// so the choice between two parabolas at x is the true one unless their values
// there are closer than eta (scan_eta below): rounding can only swap
// near-ties.  Hence, with m the smallest float value at x and "near" the
// parabolas within eta of m:
//  * near values all equal: the envelope's value is m;
//  * otherwise, when no further value lies within a / 2 of m, the near
//    parabolas keep their order on the envelope's stack whatever the others
//    do (every intersection with another one lies clearly to one side of x),
//    so replaying the reference's pushes and pops on them alone gives its
//    choice;
//  * otherwise (rare) the line is flagged for the whole float envelope.
// m needs only the positions with a d^2 <= m + a / 2: the scan runs outward
// from x, all lanes together, until that holds for every lane.  Where eta is the
// larger one the line is flagged as well.  On a periodic
// line a voxel whose m reaches the squared distance to a line end may depend
// on the imported hulls: the line is flagged for its end segments.
//
// Lines are staged in shared memory: a thread's serial float envelope spends
// its time waiting on dependent loads, while here every voxel is its own
// thread and bound by instruction issue (a shared-memory read and about five
// instructions per candidate).
#include <cfloat>
#include <algorithm>
#include <cmath>

#include <cooperative_groups.h>

#include "edt_internal.cuh"

namespace pmg {

constexpr int kScanWarps = 8;

// Values at x closer than this may be ordered either way by the reference's
// float intersections (R: distance within which near parabolas lie).
__device__ __forceinline__ float scan_eta(float a, float m, float R, float x)
{
    return a * (2.0f * R + 1.0f) * (7.0f * R + 3.0f * x + 8.0f) * 1.8e-7f + m * 4e-7f;
}

// The near parabolas of position x pushed in order as update_hull does
// (_distance.hpp:89-112), then the reference's evaluation at x.  Returns false
// when the line has to be replayed.
template <int S>
__device__ __noinline__ bool scan_resolve(const float *line, int n, int x, float a, float m, float R, float eta,
                                          float &out)
{
    if (0.25f < (3.0f * R + 1.0f) * (7.0f * R + 3.0f * (float)x + 8.0f) * 2.4e-7f)
        return false;
    constexpr int kNear = 8;
    int v[kNear];
    float f[kNear], r[kNear];
    int cnt = 0, seen = 0;
    const float top = m + 0.5f * a;
    const int D = (int)__fsqrt_rn(top / a) + 1;
    for (int q = max(0, x - D); q <= min(n - 1, x + D); q++) {
        const float dx = (float)(q - x), fq = line[S * q];
        const float val = fadd(fmul(a, fmul(dx, dx)), fq);
        if (val <= m + eta) {
            if (++seen > kNear)
                return false;
            float s = -INFINITY;
            if (cnt > 0) {
                s = isect(fq, (float)q, f[cnt - 1], (float)v[cnt - 1], a);
                while (cnt > 1 && s <= r[cnt - 1]) {
                    cnt--;
                    s = isect(fq, (float)q, f[cnt - 1], (float)v[cnt - 1], a);
                }
            }
            v[cnt] = q;
            f[cnt] = fq;
            r[cnt] = s;
            cnt++;
        } else if (val <= top) {
            return false;
        }
    }
    int k = 0;
    while (k + 1 < cnt && r[k + 1] < (float)x)
        k++;
    const float dx = (float)(x - v[k]);
    out = fadd(fmul(a, fmul(dx, dx)), f[k]);
    return true;
}

// The smallest value m and the next larger one m2, updated with the values of
// positions x - d and x + d.
__device__ __forceinline__ void scan_pair(float v0, float v1, float &m, float &m2)
{
    const float lo = fminf(v0, v1), hi = fmaxf(v0, v1), t = fmaxf(lo, m);
    m = fminf(lo, m);
    m2 = fminf(m2, fminf(hi == m ? INFINITY : hi, t == m ? INFINITY : t));
}

// One voxel per lane: the value and its line's flag bits.  line: the staged
// line (position v at line[S v]); a lane past the line's end (not live) reads
// at the last position; safe: with safe > 0 every lane's x - safe and x + safe
// lie inside the line.
template <int S>
__device__ __forceinline__ float scan_voxel(const float *line, int n, int x, int safe, bool live, float a, float inv_a,
                                            int periodic, float vcap, unsigned &need)
{
    x = min(x, n - 1);
    const float *c = line + S * x;
    float m = *c, m2 = INFINITY;
    const float half = 0.5f * a;
    int d = 1;
    bool open = true;
    // two distances per step while both sides lie inside the line
    for (const float *l = c - S, *r = c + S; d + 1 <= safe; d += 2, l -= 2 * S, r += 2 * S) {
        const float ad = fmul(a, (float)(d * d));
        open = __any_sync(0xffffffffu, live && ad <= fminf(m + half, vcap));
        if (!open)
            break;
        const float ae = fmul(a, (float)((d + 1) * (d + 1)));
        scan_pair(fadd(ad, l[0]), fadd(ad, r[0]), m, m2);
        scan_pair(fadd(ae, l[-S]), fadd(ae, r[S]), m, m2);
    }
    // near a line end, one distance at a time
    for (; open && d < n; d++) {
        const float ad = fmul(a, (float)(d * d));
        if (!__any_sync(0xffffffffu, live && ad <= fminf(m + half, vcap)))
            break;
        const float v0 = x - d >= 0 ? fadd(ad, line[S * (x - d)]) : INFINITY;
        const float v1 = x + d < n ? fadd(ad, line[S * (x + d)]) : INFINITY;
        scan_pair(v0, v1, m, m2);
    }
    if (!live || m > vcap)
        return m;
    if (m >= FLT_MAX) { // no solid voxel on the line
        need |= periodic ? kScanEnds : 0u;
        return m;
    }
    const float R = fminf(__fsqrt_rn(m * inv_a), (float)n); // (no parabola is farther)
    const float eta = scan_eta(a, m, R, (float)x);
    if (periodic) {
        const int e = min(x + 1, n - x);
        if (m + eta >= fmul(a, (float)e * (float)e)) {
            need |= kScanEnds;
            return m;
        }
    }
    // (the scan ends at m + a / 2: from about 300 voxels on long lines a parabola
    // between there and m + eta may not have been looked at)
    if (eta > half) {
        need |= kScanWhole;
        return m;
    }
    if (m2 <= m + eta) {
        float v = m;
        if (scan_resolve<S>(line, n, x, a, m, R, eta, v))
            return v;
        need |= kScanWhole;
    }
    return m;
}

// Strided lines (axis 0 or 1): one block per 32 adjacent lines, warp w on
// positions w, w + 8, ...
__global__ void __launch_bounds__(32 * kScanWarps) k_scan_cols(const float *__restrict__ fin, float *__restrict__ fout,
                                                               Lines Ls, float a, float inv_a, int periodic, int form,
                                                               MorphEpi me, float vcap, uint8_t *__restrict__ flag,
                                                               const int *__restrict__ wide)
{
    if (blockIdx.x >= kFirstBlocks && left_to_envelope(wide))
        return;
    extern __shared__ float s_line[]; // [n][32]
    __shared__ unsigned s_need[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int tiles = (Ls.nb2 + 31) / 32;
    const int ra = blockIdx.x / tiles, kb = (blockIdx.x - ra * tiles) * 32 + lane;
    const bool live = kb < Ls.nb2;
    const long long li = (long long)ra * Ls.nb2 + (live ? kb : 0);
    const LineGeo g = line_addr(Ls, li);
    const int n = g.n;
    const float *src = fin + g.base;
    if (threadIdx.x < 32)
        s_need[threadIdx.x] = 0;
    bool some = false;
#pragma unroll 8
    for (int x = w; x < n; x += kScanWarps) {
        const float v = __ldg(src + x * g.stride);
        some |= v < FLT_MAX;
        s_line[x * 32 + lane] = v;
    }
    // without a solid on any of the lines, nothing to scan
    const bool scan = __syncthreads_or(some) || periodic;
    if (blockIdx.x < kFirstBlocks && left_to_envelope(wide))
        return;
    unsigned need = 0;
    for (int x = w; x < n; x += kScanWarps) {
        const float v = scan ? scan_voxel<32>(s_line + lane, n, x, min(x, n - 1 - x), live, a, inv_a, periodic, vcap, need)
                             : FLT_MAX;
        if (!live)
            continue;
        if (form == PMG_EDT_MORPH)
            morph_store(me, g, x, v);
        else
            fout[g.base + x * g.stride] = form == PMG_EDT_DIST ? __fsqrt_rn(v) : v;
    }
    if (need)
        atomicOr(s_need + lane, need);
    __syncthreads();
    if (w == 0 && live)
        flag[li] = (uint8_t)s_need[lane];
}

// Contiguous lines: one warp per row, lanes on 32 consecutive positions.
__global__ void __launch_bounds__(32 * kScanWarps) k_scan_rows(const float *__restrict__ fin, float *__restrict__ fout,
                                                               Lines Ls, float a, float inv_a, int periodic, int form,
                                                               MorphEpi me, float vcap, uint8_t *__restrict__ flag,
                                                               const int *__restrict__ wide)
{
    if (blockIdx.x >= kFirstBlocks && left_to_envelope(wide))
        return;
    bool early = blockIdx.x < kFirstBlocks;
    extern __shared__ float s_line[]; // [kScanWarps][n]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long nlines = Ls.count();
    const int n = (int)Ls.s2;
    float *row = s_line + (long long)w * n;
    for (long long li = blockIdx.x * (long long)kScanWarps + w; li < nlines;
         li += (long long)gridDim.x * kScanWarps) {
        const LineGeo g = line_addr(Ls, li);
        const float *src = fin + g.base;
        bool some = false;
#pragma unroll 8
        for (int x = lane; x < n; x += 32) {
            const float v = __ldg(src + x);
            some |= v < FLT_MAX;
            row[x] = v;
        }
        const bool scan = __any_sync(0xffffffffu, some) || periodic;
        __syncwarp();
        if (early && left_to_envelope(wide))
            return;
        early = false;
        unsigned need = 0;
        for (int x0 = 0; x0 < n; x0 += 32) {
            const int x = x0 + lane;
            const bool live = x < n;
            const float v = scan ? scan_voxel<1>(row, n, x, min(x0, n - 32 - x0), live, a, inv_a, periodic, vcap, need)
                                 : FLT_MAX;
            if (!live)
                continue;
            if (form == PMG_EDT_MORPH)
                morph_store(me, g, x, v);
            else
                fout[g.base + x] = form == PMG_EDT_DIST ? __fsqrt_rn(v) : v;
        }
        need = __reduce_or_sync(0xffffffffu, need);
        if (lane == 0)
            flag[li] = (uint8_t)need;
        __syncwarp();
    }
}

// Wide pores.  A scan's cost grows with the distances of its voxels, the float
// envelope's hardly does, so a probe in front of the pass estimates the steps of
// a scan from kProbeGroups of its warps (32 adjacent lines, or 32 consecutive
// positions of a row) and sets *wide when the envelope is the cheaper one.
// One cluster, so that the sum needs no clearing.
constexpr int kProbeBlocks = 8, kProbeThreads = 512, kProbeGroups = kProbeBlocks * kProbeThreads / 32;

__global__ void __cluster_dims__(kProbeBlocks, 1, 1) __launch_bounds__(kProbeThreads)
    k_pore_probe(const float *__restrict__ fin, Lines Ls, float a, float inv_a, float vcap, float most, float budget,
                 int *wide)
{
    cudaTriggerProgrammaticLaunchCompletion(); // (the pass may start: its first blocks wait)
    __shared__ unsigned s_sum;
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        s_sum = 0;
    __syncthreads();
    // group q of equal shares of the lines; where in its share and along the
    // lines by multiplicative hashes (a regular pattern could follow the axes)
    const unsigned q = blockIdx.x * (kProbeThreads / 32) + (threadIdx.x >> 5);
    const long long nl = Ls.count(), li = (q * nl + (long long)(q * 2246822519u >> 4) % nl) / kProbeGroups;
    LineGeo g = line_addr(Ls, Ls.ax == 2 ? li : min(li + lane, nl - 1));
    const int n = g.n;
    int x = (int)((q * 2654435761u >> 8) % (unsigned)n);
    if (Ls.ax == 2)
        x = min(x / 32 * 32 + lane, n - 1);
    const float *c = fin + g.base;
    float m = c[x * g.stride];
    const auto at = [&](int d) {
        m = fminf(m, fminf(c[max(x - d, 0) * g.stride], c[min(x + d, n - 1) * g.stride]) + a * (float)(d * d));
    };
    // every distance up to 128 (lines of a volume that is thin along the earlier axes
    // hold solids at single positions), then some
    int d = 0;
    bool open = true;
    for (; d < 128 && open; d += 16) {
#pragma unroll
        for (int u = 1; u <= 16; u++)
            at(d + u);
        open = __any_sync(0xffffffffu, m > a * (float)((d + 16) * (d + 16)));
    }
    for (; open && d < n; d += d / 2) {
#pragma unroll
        for (int u = 1; u <= 4; u++)
            at(d + d * u / 8);
        open = __any_sync(0xffffffffu, m > a * (float)(d * d / 4 * 9));
    }
    // (a warp scans as far as its farthest lane; lines that a scan would leave to the
    // envelope after all count as far)
    const float R = fminf(__fsqrt_rn(m * inv_a), (float)n);
    const bool whole = m <= vcap && scan_eta(a, m, R, (float)x) > 0.5f * a;
    const unsigned far = __reduce_max_sync(0xffffffffu, (unsigned)(whole ? most : fminf(R, most)));
    if (lane == 0)
        atomicAdd(&s_sum, far);
    cluster.sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned sum = 0;
        for (int k = 0; k < kProbeBlocks; k++)
            sum += *cluster.map_shared_rank(&s_sum, k);
        *wide = (float)sum > budget * (float)kProbeGroups;
    }
    cluster.sync(); // (the other blocks' sums are read until here)
}

// Steps a voxel from which the envelope is the faster one.  A step costs about 1 ps a
// voxel (512^3: 0.14 ms a pass), the envelope 15 to 50 ps (1.9 to 7 ms) and at least
// one chain of n pushes (1 to 2 us each), hence the term in the lines.  With few lines
// a scan is a chain too: of columns n / 8 rounds of as many steps as their
// distances (65 ns each), of rows n / 32, hence the upper ends.  Scan alone,
// envelope alone, chosen, in ms, voxels of 2.25: 512^3 field of sigma 4: 2.0, 5.1, 2.0;
// cavity of radius 230: 7.2, 5.1, 5.1; points 20 voxels apart on average: 51, 10.6, 10.6;
// 256^3 points 10 voxels apart: 1.97, 1.39, 1.1; one pass of 1000 x 1000, points 40, 80
// voxels apart: 0.46, 0.91, 0.46 and 2.15, 1.01, 1.01; 1024 x 100, points 20: 0.25, 0.95, 0.25.
// On periodic lines the ends are replayed after a scan, so the crossing lies lower
// (voxels 1 x 1 x 2, 512^3 field of sigma 4: 3.5, 5.5, 3.5; sigma 20: 12.7, 8.6, 8.6; 1000 x
// 1000, points 4 and 20 voxels apart: 0.90, 2.3, 0.90 and 3.9, 3.8, 3.8).
static float scan_budget(const Lines &Ls, int periodic)
{
    const float nl = (float)Ls.count();
    const int k = tune_value(kTuneEdtWide); // 1024: as it is; 0: always the envelope, 8193: never
    if (k == 0)
        return -1.0f;
    if (k > 8192)
        return INFINITY;
    const float steps = periodic ? std::min(12.0f, std::max(5.0f, 0.11e6f / nl))
                                 : std::min(Ls.ax == 2 ? 190.0f : 95.0f, std::max(36.0f, 1.3e6f / nl));
    return steps * ((float)k / 1024.0f);
}

// *choice = wide once the probe has set it, null where no scan of the pass can
// take more steps than the budget (short lines, a small cap).
int launch_pore_probe(const float *fin, const Lines &Ls, float res, float vcap, int periodic, int *wide,
                      const int **choice, cudaStream_t st)
{
    const float a = res * res, inv_a = 1.0f / a;
    const int n = (int)(Ls.ax == 0 ? Ls.s0 : Ls.ax == 1 ? Ls.s1 : Ls.s2);
    // the most steps of a voxel: to the line's end, or to the cap
    const float most = std::fmin((float)n, std::sqrt(vcap * inv_a) + 1.0f), budget = scan_budget(Ls, periodic);
    *choice = nullptr;
    // (on a small volume with short lines the two lie close together whatever the
    // distances: 100 x 300 x 100, rows without a solid nearby, 0.40 and 0.11 ms, where
    // the probe is 2 to 5 us of calls from 70)
    if (most <= budget || (!periodic && budget >= 0.0f && n <= 128 && (float)Ls.count() * (float)n < 5e6f))
        return PMG_OK;
    const int ps__ = prof_begin("k_pore_probe", st);
    k_pore_probe<<<kProbeBlocks, kProbeThreads, 0, st>>>(fin, Ls, a, inv_a, vcap, most, budget, wide);
    prof_end(ps__, 0.0, st);
    PMG_CHECK_LAUNCH();
    *choice = wide;
    return PMG_OK;
}

int launch_scan(const float *fin, float *fout, const Lines &Ls, float res, const pmg_axis_cfg &cfg, int form,
                const MorphEpi &me, float vcap, uint8_t *flag, const int *wide, cudaStream_t st)
{
    const float a = res * res, inv_a = 1.0f / a;
    const int per = cfg.periodic ? 1 : 0;
    if (Ls.ax == 2) {
        const size_t smem = sizeof(float) * (size_t)kScanWarps * (size_t)Ls.s2;
        const int ps__ = prof_begin("k_scan_rows", st);
        const unsigned grid = grid_for(Ls.count(), kScanWarps, 152LL * 64);
        if (wide)
            PMG_CUDA(launch_after_probe(k_scan_rows, dim3(grid), 32 * kScanWarps, smem, st, fin, fout, Ls, a, inv_a, per, form, me,
                                        vcap, flag, wide));
        else
            k_scan_rows<<<grid, 32 * kScanWarps, smem, st>>>(fin, fout, Ls, a, inv_a, per, form, me, vcap, flag, wide);
        prof_end(ps__, (double)Ls.count() * Ls.s2 * (form == PMG_EDT_MORPH ? 5 : 8), st);
    } else {
        const int n = (int)(Ls.ax == 0 ? Ls.s0 : Ls.s1);
        const size_t smem = sizeof(float) * 32 * (size_t)n;
        if (smem > 47 * 1024)
            PMG_CUDA(cudaFuncSetAttribute(k_scan_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const long long blocks = (long long)Ls.nb1 * ((Ls.nb2 + 31) / 32);
        const int ps__ = prof_begin("k_scan_cols", st);
        if (wide)
            PMG_CUDA(launch_after_probe(k_scan_cols, dim3((unsigned)blocks), 32 * kScanWarps, smem, st, fin, fout, Ls, a, inv_a, per,
                                        form, me, vcap, flag, wide));
        else
            k_scan_cols<<<(unsigned)blocks, 32 * kScanWarps, smem, st>>>(fin, fout, Ls, a, inv_a, per, form, me, vcap, flag,
                                                                        wide);
        prof_end(ps__, (double)Ls.count() * n * (form == PMG_EDT_MORPH ? 5 : 8), st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

} // namespace pmg
