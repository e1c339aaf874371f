// Porosimetry and morphological drainage driven from native code.
//
// porosimetry (src/pmmoto/filters/porosimetry.py:84-160, mode="distance"):
//   erode -> [inlet-connected] -> if phase 1 exists: [multiphase constraint:
//   inlet-connected phase 1 of the multiphase image] -> dilate.
// drainage, standard method (src/pmmoto/filters/equilibrium_distribution.py:
//   25-179): per capillary pressure, porosimetry with the inlet and multiphase
//   constraints, outlet-connected wetting phase, update, reservoir refill,
//   wetting-phase count in the own region (the saturation numerator).
// All images stay on the device between steps.  A drainage reads back its
// per-pressure counts at the end; per pressure it waits only where a branch on the
// host depends on the data (porosimetry's phase counts without a growing
// selection, the seed count of a dilation by scan).
#include <algorithm>
#include <cmath>
#include <vector>

#include "edt_internal.cuh"
#include "pmg_internal.cuh"

namespace pmg {

// Bytes equal to 1 in both words -> 1, else 0 (four voxels per 32-bit word).
__device__ __forceinline__ uint32_t both_one(uint32_t a, uint32_t b)
{
    const uint32_t z = (a ^ 0x01010101u) | (b ^ 0x01010101u);
    const uint32_t t = ((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z; // high bit set where the byte is nonzero
    return (~t & 0x80808080u) >> 7;
}

// res = (res == 1 && nconn == 1) ? 1 : 0, i.e. where((res != 1) | (nconn != 1), 0, res)
__global__ void k_constrain(uint8_t *res, const uint8_t *__restrict__ nconn, long long n)
{
    const long long nw = n >> 4; // 16-byte vectors (both buffers are 256-byte aligned)
    uint4 *r4 = (uint4 *)res;
    const uint4 *c4 = (const uint4 *)nconn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nw;
         q += (long long)gridDim.x * blockDim.x) {
        uint4 a = r4[q];
        const uint4 b = c4[q];
        a.x = both_one(a.x, b.x);
        a.y = both_one(a.y, b.y);
        a.z = both_one(a.z, b.z);
        a.w = both_one(a.w, b.w);
        r4[q] = a;
    }
    for (long long i = (nw << 4) + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        res[i] = (res[i] == 1 && nconn[i] == 1) ? 1 : 0;
}

// Erosion by thresholding a precomputed squared EDT (subtraction's
// np.where(d <= r, 0, 1), unpad being the identity without extension), wall
// planes forced to 0 (set_wall_bcs).  One warp per (i, j) row.
struct ErodeThr {
    float lim; // within_limit of the radius
    int wall[6];
};

// Rows of a volume inside an extended one: the first voxel at lo.
struct ExtRows {
    long long X1, X2, lo0, lo1, lo2;
    __device__ __forceinline__ long long row(long long i, long long j) const
    {
        return ((i + lo0) * X1 + j + lo1) * X2 + lo2;
    }
};

__global__ void k_erode_from_edt(const float *__restrict__ D, uint8_t *__restrict__ out, long long s0,
                                 long long s1, long long s2, ErodeThr T, ExtRows X)
{
    const long long rows = s0 * s1;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = warp; r < rows; r += nwarps) {
        const long long i = r / s1, j = r - (r / s1) * s1;
        const bool wrow = (T.wall[0] && i == 0) || (T.wall[1] && i == s0 - 1) || (T.wall[2] && j == 0) ||
                          (T.wall[3] && j == s1 - 1);
        const long long base = r * s2;
        const float *src = D + X.row(i, j);
#pragma unroll 4
        for (long long k = lane; k < s2; k += 32) {
            uint8_t o = src[k] <= T.lim ? 0 : 1;
            if (wrow || (T.wall[4] && k == 0) || (T.wall[5] && k == s2 - 1))
                o = 0;
            out[base + k] = o;
        }
    }
}

struct Work {
    uint8_t *t1, *t2, *t3; // uint8 volumes
    uint8_t *E;            // morphology scratch
    float *A, *B;
    int *P;
    uint8_t *M, *mark; // per-block masks and marks of the binary selection
    unsigned *rows;    // row words (a drainage's selection)
    int *err;
    unsigned long long *cnt; // scalar counter
    void *base;
};

static int work_alloc(Work &w, const int64_t *shape, size_t morph_bytes, cudaStream_t st)
{
    const size_t n = (size_t)shape[0] * shape[1] * shape[2];
    const size_t a = (n + 255) & ~(size_t)255;
    const size_t nb = (size_t)((shape[0] + 1) / 2) * ((shape[1] + 1) / 2) * ((shape[2] + 1) / 2);
    const size_t bb = (nb + 255) & ~(size_t)255;
    const size_t rb = rows_bytes(shape);
    const size_t total = 3 * a + ((morph_bytes + 255) & ~(size_t)255) + a * 4 + 2 * bb + rb + 512;
    PMG_TRY(scratch_alloc(&w.base, total, st));
    char *p = (char *)w.base;
    w.t1 = (uint8_t *)p;
    p += a;
    w.t2 = (uint8_t *)p;
    p += a;
    w.t3 = (uint8_t *)p;
    p += a;
    w.E = (uint8_t *)p;
    p += (morph_bytes + 255) & ~(size_t)255;
    w.P = (int *)p;
    p += a * 4;
    w.M = (uint8_t *)p;
    p += bb;
    w.mark = (uint8_t *)p;
    p += bb;
    w.rows = (unsigned *)p;
    p += rb;
    w.err = (int *)p;
    w.cnt = (unsigned long long *)(p + 256);
    return PMG_OK;
}

// Step of every voxel in a growing eroded space: the first radius index whose
// threshold its capped squared distance exceeds (the thresholds never rise),
// read from a table over the capped values; wall planes never enter (255).
// One warp per (i, j) row.
__global__ void k_step_volume(const uint16_t *__restrict__ KC, uint8_t *__restrict__ S,
                              const uint8_t *__restrict__ tab, int tmax, long long s0, long long s1, long long s2,
                              unsigned walls)
{
    __shared__ uint8_t s_tab[kCapMaxT + 2];
    for (int v = threadIdx.x; v <= tmax; v += blockDim.x)
        s_tab[v] = tab[v];
    __syncthreads();
    const long long rows = s0 * s1;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = warp; r < rows; r += nwarps) {
        const long long i = r / s1, j = r - (r / s1) * s1;
        const bool wrow = ((walls & 1u) && i == 0) || ((walls & 2u) && i == s0 - 1) || ((walls & 4u) && j == 0) ||
                          ((walls & 8u) && j == s1 - 1);
        const long long base = r * s2;
        for (long long k = lane; k < s2; k += 32) {
            const int v = min((int)KC[base + k], tmax);
            const bool wall = wrow || ((walls & 16u) && k == 0) || ((walls & 32u) && k == s2 - 1);
            S[base + k] = wall ? (uint8_t)255 : s_tab[v];
        }
    }
}

// ... of any voxel size, from the float distances: the first radius at which the
// erosion (k_erode_from_edt's comparison) keeps the voxel.  The limits never
// rise, so a bisection finds it; step: the radius index of each limit.
// Bound by the four bytes read and one written per voxel: 20 erosions written
// and labelled again took 2.0 of 5.6 ms of a 150 x 121 x 99 drainage.
__global__ void k_step_volume_f32(const float *__restrict__ D, uint8_t *__restrict__ S,
                                  const float *__restrict__ thr, const uint8_t *__restrict__ step, int nthr,
                                  long long s0, long long s1, long long s2, unsigned walls)
{
    __shared__ float s_thr[256];
    __shared__ uint8_t s_step[256];
    for (int v = threadIdx.x; v < nthr; v += blockDim.x) {
        s_thr[v] = thr[v];
        s_step[v] = step[v];
    }
    __syncthreads();
    const long long rows = s0 * s1;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = warp; r < rows; r += nwarps) {
        const long long i = r / s1, j = r - (r / s1) * s1;
        const bool wrow = ((walls & 1u) && i == 0) || ((walls & 2u) && i == s0 - 1) || ((walls & 4u) && j == 0) ||
                          ((walls & 8u) && j == s1 - 1);
        const long long base = r * s2;
        for (long long k = lane; k < s2; k += 32) {
            const float d = D[base + k];
            int lo = 0, hi = nthr; // the first limit below d (none: nthr)
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (d <= s_thr[mid])
                    lo = mid + 1;
                else
                    hi = mid;
            }
            const bool wall = wrow || ((walls & 16u) && k == 0) || ((walls & 32u) && k == s2 - 1);
            S[base + k] = wall || lo == nthr ? (uint8_t)255 : s_step[lo];
        }
    }
}

static void morph_split(Work &w, const int64_t *shape, const int32_t *bc, const int32_t *ext,
                        uint8_t *&E, float *&A, float *&B)
{
    long long nv = 1;
    for (int d = 0; d < 3; d++)
        nv *= shape[d] + (bc[2 * d] == PMG_BC_PERIODIC ? ext[2 * d] + ext[2 * d + 1] : 0);
    E = w.E;
    A = (float *)(w.E + (((size_t)nv + 255) & ~(size_t)255));
    B = A + nv;
}

static int count_sync(const uint8_t *img, const int64_t *shape, const int64_t *box, uint8_t value, Work &w,
                      cudaStream_t st, long long &out)
{
    PMG_CUDA(cudaMemsetAsync(w.cnt, 0, sizeof(unsigned long long), st));
    PMG_TRY(count_eq_async(img, shape, box, value, w.cnt, st));
    unsigned long long h = 0;
    PMG_CUDA(cudaMemcpyAsync(&h, w.cnt, sizeof(h), cudaMemcpyDeviceToHost, st));
    PMG_CUDA(cudaStreamSynchronize(st));
    out = (long long)h;
    return PMG_OK;
}

// A second stream that takes work between begin (after what the first stream
// holds) and end, which join makes the first stream wait for.
struct Fork {
    cudaStream_t side = nullptr;
    cudaEvent_t from = nullptr, to = nullptr;
    bool pending = false;
    int open()
    {
        PMG_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        PMG_CUDA(cudaEventCreateWithFlags(&from, cudaEventDisableTiming));
        PMG_CUDA(cudaEventCreateWithFlags(&to, cudaEventDisableTiming));
        return PMG_OK;
    }
    int begin(cudaStream_t st)
    {
        PMG_CUDA(cudaEventRecord(from, st));
        PMG_CUDA(cudaStreamWaitEvent(side, from, 0));
        return PMG_OK;
    }
    int end()
    {
        if (cudaEventRecord(to, side) != cudaSuccess) {
            cudaStreamSynchronize(side); // (what it holds must not outlive its scratch)
            set_error("drainage: event record failed");
            return PMG_ECUDA;
        }
        pending = true;
        return PMG_OK;
    }
    int join(cudaStream_t st)
    {
        if (pending)
            PMG_CUDA(cudaStreamWaitEvent(st, to, 0));
        pending = false;
        return PMG_OK;
    }
    ~Fork()
    {
        // (work still queued is finished before the stream goes)
        if (to)
            cudaEventDestroy(to);
        if (from)
            cudaEventDestroy(from);
        if (side)
            cudaStreamDestroy(side);
    }
};

// porosimetry.py:84-160 (mode="distance") into `out`.
static int porosimetry_run(const uint8_t *pm, uint8_t *out, const int64_t *shape, const int32_t *bc,
                           const int32_t *pad, const int32_t *ext_e, const int32_t *ext_d, const float *res,
                           double r_e, int cmp_e, double r_d, int cmp_d, int inlet, const uint8_t *mp,
                           const Boxes &Bx, Work &w, cudaStream_t st, double ball_e, double ball_d,
                           const float *De = nullptr, const uint16_t *KC = nullptr, int Te = -1,
                           bool m1_counted = false, GrowSel *g_er = nullptr, GrowSel *g_nw = nullptr,
                           int *orange = nullptr, unsigned *rows_out = nullptr, Fork *eroded = nullptr)
{
    // a drainage: rows_out, the result as row words (out is then scratch); eroded,
    // where the eroded space's marks of this radius were made
    // m1_counted: w.cnt[1] already holds count(mp == 1) (the drainage update
    // counts it); the inlet selection counts its kept voxels into w.cnt[0], and
    // both come back with one copy
    const long long n = shape[0] * shape[1] * shape[2];
    const int64_t all[6] = {0, shape[0], 0, shape[1], 0, shape[2]};
    uint8_t *E;
    float *A, *B;
    morph_split(w, shape, bc, ext_e, E, A, B);
    uint8_t *cur = w.t1;
    if (eroded) {
        // both selections grow along the curve: one pass writes the eroded
        // inlet-connected space constrained by the inlet-connected
        // non-wetting phase (when that phase exists, counted in w.cnt[1])
        PMG_TRY(grow_marks_phase(*g_nw, mp, 1, shape, bc, pad, Bx.inlet, w.err, st));
        PMG_TRY(eroded->join(st));
        // the selection's x range (w.cnt[4]) limits the dilation to the planes
        // it can reach; the dilation's result range goes to orange.  Like the
        // kept count (w.cnt[0]) it is zero here (DrainCounts)
        int *xr = (int *)(w.cnt + 4);
        // the selection is written as row words (w.rows): the dilation's row
        // pass reads them directly (w.t2 receives bytes on other paths)
        PMG_TRY(grow_pair_select(*g_er, *g_nw, w.cnt + 1, w.rows, shape, w.err, st, w.cnt, xr));
        PMG_TRY(eroded->begin(st)); // the next radius's marks may follow
        // the dilation reads the kept count (w.cnt[0]) on the device: no
        // dilation of an empty selection, and no host round trip per radius
        morph_split(w, shape, bc, ext_d, E, A, B);
        return morph_run(w.t2, out, shape, bc, pad, ext_d, res, r_d, cmp_d, 1, E, A, B, st, ball_d, w.cnt, xr,
                         orange, w.rows, rows_out);
    }
    PMG_CUDA(cudaMemsetAsync(w.cnt, 0, sizeof(unsigned long long), st));
    if (orange) {
        // the paths below write the whole result
        k_set_int2<<<1, 32, 0, st>>>(orange, 0, (int)shape[0] - 1);
        PMG_CHECK_LAUNCH();
    }
    if (KC && inlet) {
        PMG_TRY(select_run_erode(KC, Te, w.t2, shape, bc, pad, Bx.inlet, nullptr, PMG_SEL_INLET, w.P, w.M, w.mark,
                                 w.err, st, w.cnt));
        cur = w.t2;
    } else if (De) {
        ErodeThr T;
        T.lim = within_limit(r_e, cmp_e, ball_e);
        for (int q = 0; q < 6; q++)
            T.wall[q] = bc[q] == PMG_BC_WALL;
        const int ps__ = prof_begin("k_erode_from_edt", st);
        k_erode_from_edt<<<grid_for(shape[0] * shape[1] * 32, 256, 152LL * 64), 256, 0, st>>>(
            De, w.t1, shape[0], shape[1], shape[2], T, ExtRows{shape[1], shape[2], 0, 0, 0});
        prof_end(ps__, (double)n * 5, st);
        PMG_CHECK_LAUNCH();
    } else {
        PMG_TRY(morph_run(pm, w.t1, shape, bc, pad, ext_e, res, r_e, cmp_e, 0, E, A, B, st, ball_e));
    }
    if (inlet && cur == w.t1) {
        // the eroded image holds only 0 and 1
        PMG_TRY(select_run_binary(w.t1, w.t2, 1, shape, bc, pad, Bx.inlet, nullptr, PMG_SEL_INLET, -1, w.P, w.M,
                                  w.mark, w.err, st, w.cnt));
        cur = w.t2;
    }
    long long c1 = 0, m1 = -1;
    if (inlet) {
        unsigned long long h[2] = {0, 0};
        PMG_CUDA(cudaMemcpyAsync(h, w.cnt, sizeof(h), cudaMemcpyDeviceToHost, st));
        PMG_CUDA(cudaStreamSynchronize(st));
        c1 = (long long)h[0];
        if (m1_counted)
            m1 = (long long)h[1];
    } else {
        PMG_TRY(count_sync(cur, shape, all, 1, w, st, c1));
    }
    if (c1 > 0) {
        if (mp) {
            if (m1 < 0)
                PMG_TRY(count_sync(mp, shape, all, 1, w, st, m1));
            if (m1 > 0) {
                if (g_nw)
                    PMG_TRY(select_grow_binary(*g_nw, mp, 1, w.t3, shape, bc, pad, Bx.inlet, nullptr,
                                               PMG_SEL_INLET, w.err, st));
                else
                    PMG_TRY(select_run_binary(mp, w.t3, 1, shape, bc, pad, Bx.inlet, nullptr, PMG_SEL_INLET, 1,
                                              w.P, w.M, w.mark, w.err, st));
                {
                    const int ps__ = prof_begin("k_constrain", st);
                    k_constrain<<<grid_for(n / 16 + 1, 256, 152LL * 32), 256, 0, st>>>(cur, w.t3, n);
                    prof_end(ps__, (double)n * 3, st);
                }
                PMG_CHECK_LAUNCH();
            }
        }
        morph_split(w, shape, bc, ext_d, E, A, B);
        PMG_TRY(morph_run(cur, out, shape, bc, pad, ext_d, res, r_d, cmp_d, 1, E, A, B, st, ball_d, nullptr, nullptr,
                          nullptr, nullptr, rows_out));
    } else if (rows_out) {
        PMG_TRY(bytes_to_rows(cur, rows_out, shape, st));
    } else if (cur != out) {
        PMG_CUDA(cudaMemcpyAsync(out, cur, (size_t)n, cudaMemcpyDeviceToDevice, st));
    }
    return PMG_OK;
}

// ---- pore size distribution ---------------------------------------------------------
// Voxels whose shared erosion distance lies too close to a radius's threshold
// for its decision to be the one of that radius's own distances (pmg_pore_sizes
// below): flag[k] of threshold k.  thr: squared thresholds; top: clear of all of them; a1, a2, x1, x2: squared
// spacings and extended lengths of the two envelope passes.
__global__ void k_near_thresholds(const float *__restrict__ D, long long s0, long long s1, long long s2, ExtRows X,
                                  const float *__restrict__ thr, int nthr, float top, float a1, float x1, float a2,
                                  float x2, int *flag)
{
    const long long rows = s0 * s1;
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; r < rows; r += nwarps) {
        const float *src = D + X.row(r / s1, r % s1);
        for (long long k = lane; k < s2; k += 32) {
            const float v = src[k];
            if (v > top)
                continue;
            const float R1 = sqrtf(v / a1), R2 = sqrtf(v / a2);
            const float band = 3.6e-7f * (a1 * (2.0f * R1 + 1.0f) * (7.0f * R1 + 3.0f * x1 + 8.0f) +
                                          a2 * (2.0f * R2 + 1.0f) * (7.0f * R2 + 3.0f * x2 + 8.0f)) +
                               4e-6f * v;
            // (every lane the same threshold: a bisection's loads depend on each
            // other and took 2.2 ms instead of 0.22 ms for 25 at 200^3)
            for (int q = 0; q < nthr; q++)
                if (fabsf(v - thr[q]) <= band)
                    flag[q] = 1;
        }
    }
}

// todo = 1 at the pore voxels (pm == 1).
__global__ void k_pore_mask(const uint8_t *__restrict__ pm, uint8_t *__restrict__ todo, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        todo[i] = pm[i] == 1;
}

// The radius at the voxels to do that this opening (0 / 1) covers; they are done
// then, unless the radius is zero (such a size counts as none).  Sixteen voxels
// per thread; bound by the two bytes read per voxel.  Reading the sizes
// themselves took 19 us at 200^3.
__global__ void k_first_cover(const uint8_t *__restrict__ cover, uint8_t *__restrict__ todo, double *__restrict__ out,
                              double radius, long long n)
{
    const long long step = (long long)gridDim.x * blockDim.x, n16 = n >> 4;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n16; q += step) {
        const uint4 c = reinterpret_cast<const uint4 *>(cover)[q];
        uint4 t = reinterpret_cast<const uint4 *>(todo)[q];
        const unsigned hit[4] = {c.x & t.x, c.y & t.y, c.z & t.z, c.w & t.w};
        if (!(hit[0] | hit[1] | hit[2] | hit[3]))
            continue;
#pragma unroll
        for (int w = 0; w < 4; w++)
            for (unsigned h = hit[w]; h; h &= h - 1)
                out[16 * q + 4 * w + ((__ffs(h) - 1) >> 3)] = radius;
        if (radius != 0.0)
            reinterpret_cast<uint4 *>(todo)[q] =
                make_uint4(t.x & ~hit[0], t.y & ~hit[1], t.z & ~hit[2], t.w & ~hit[3]);
    }
    for (long long i = 16 * n16 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += step)
        if (cover[i] & todo[i]) {
            out[i] = radius;
            if (radius != 0.0)
                todo[i] = 0;
        }
}

static int ext_of(const int32_t *bc, const int32_t *pad, const int32_t *ratio, int32_t *ext)
{
    for (int d = 0; d < 3; d++)
        for (int s = 0; s < 2; s++) {
            const int b = bc[2 * d + s];
            ext[2 * d + s] = (b == PMG_BC_END || (b == PMG_BC_WALL && pad[2 * d + s] == 1)) ? 0 : ratio[d];
        }
    return PMG_OK;
}

static size_t max_morph_bytes(const int64_t *shape, const int32_t *bc, const int32_t *ext_a, const int32_t *ext_b)
{
    const size_t a = morph_scratch_bytes(shape, bc, ext_a), b = morph_scratch_bytes(shape, bc, ext_b);
    return a > b ? a : b;
}

// A failed allocation alone, whose error is then taken back.
static bool no_room(int status)
{
    if (status != PMG_ECUDA || cudaPeekAtLastError() != cudaErrorMemoryAllocation)
        return false;
    cudaGetLastError();
    return true;
}

static int check_common(const int64_t *shape, const int32_t *bc, const int32_t *pad)
{
    PMG_TRY(check_geometry(shape, bc, pad));
    return check_volume(shape);
}

} // namespace pmg

using namespace pmg;

extern "C" int pmg_porosimetry(const uint8_t *pm_img, const uint8_t *mp_img, uint8_t *out,
                               const int64_t shape[3], const int32_t bc[6], const int32_t pad[6],
                               const int64_t inlet_box[6], const float res[3], double r_erode,
                               int32_t cmp_erode, const int32_t ratio_erode[3], double r_dilate,
                               int32_t cmp_dilate, const int32_t ratio_dilate[3], int32_t inlet,
                               double ball_erode, double ball_dilate, void *stream)
{
    PMG_TRY(check_common(shape, bc, pad));
    if (!pm_img || !out || !res || !ratio_erode || !ratio_dilate) {
        set_error("pmg_porosimetry: null argument");
        return PMG_EINVAL;
    }
    cudaStream_t st = as_stream(stream);
    int32_t ext_e[6], ext_d[6];
    ext_of(bc, pad, ratio_erode, ext_e);
    ext_of(bc, pad, ratio_dilate, ext_d);
    Boxes Bx{};
    for (int q = 0; q < 6; q++) {
        Bx.inlet[q] = inlet_box ? inlet_box[q] : -1;
        Bx.outlet[q] = -1;
    }
    Work w{};
    PMG_TRY(work_alloc(w, shape, max_morph_bytes(shape, bc, ext_e, ext_d), st));
    PMG_CUDA(cudaMemsetAsync(w.err, 0, sizeof(int), st));
    int s = porosimetry_run(pm_img, out, shape, bc, pad, ext_e, ext_d, res, r_erode, cmp_erode, r_dilate,
                            cmp_dilate, inlet, mp_img, Bx, w, st, ball_erode, ball_dilate);
    if (s == PMG_OK)
        s = check_err(w.err, st);
    int s2 = scratch_free(w.base, st);
    return s != PMG_OK ? s : s2;
}

// The openings of a pore size distribution (porosimetry.py:199-227) share one
// erosion distance field where that gives every radius its own decisions.  A
// radius's own field is that of the image extended by its own reach; the field
// of the largest extension holds every seed of it and, beyond, only seeds
// farther than the radius.  What may differ is which of two parabolas within
// rounding (edt_scan.cu's eta, once per envelope pass) the reference takes, as
// positions are counted from another origin: a radius with a voxel whose
// distance lies within twice that of the threshold is eroded by itself
// (k_near_thresholds).  Isotropic power-of-two voxels have exact fields.
// 25 fields of a periodic 200^3 pack cost 11 of 13.5 ms of its kernels.
extern "C" int pmg_pore_sizes(const uint8_t *pm_img, double *out, const int64_t shape[3], const int32_t bc[6],
                              const int32_t pad[6], const int64_t inlet_box[6], const float res[3], int32_t n_radii,
                              const double *radii, const int32_t *cmp64, const int32_t *ratios,
                              const double *ball_erode, const double *ball_dilate, int32_t inlet, void *stream)
{
    PMG_TRY(check_common(shape, bc, pad));
    if (!pm_img || !out || !res || n_radii < 0 ||
        (n_radii > 0 && (!radii || !cmp64 || !ratios || !ball_erode || !ball_dilate))) {
        set_error("pmg_pore_sizes: null argument");
        return PMG_EINVAL;
    }
    cudaStream_t st = as_stream(stream);
    const long long n = shape[0] * shape[1] * shape[2];
    PMG_CUDA(cudaMemsetAsync(out, 0, (size_t)n * sizeof(double), st));
    if (n_radii == 0)
        return PMG_OK;
    Boxes Bx{};
    for (int q = 0; q < 6; q++) {
        Bx.inlet[q] = inlet_box ? inlet_box[q] : -1;
        Bx.outlet[q] = -1;
    }
    // the largest extension, and each radius's
    std::vector<int32_t> ext((size_t)n_radii * 6);
    int32_t big[6] = {0, 0, 0, 0, 0, 0};
    size_t mb = 0;
    for (int k = 0; k < n_radii; k++) {
        int32_t *e = ext.data() + 6 * (size_t)k;
        ext_of(bc, pad, ratios + 3 * k, e);
        for (int q = 0; q < 6; q++)
            big[q] = e[q] > big[q] ? e[q] : big[q];
        const size_t b = morph_scratch_bytes(shape, bc, e);
        mb = b > mb ? b : mb;
    }
    Work w{};
    PMG_TRY(work_alloc(w, shape, mb, st));
    PMG_CUDA(cudaMemsetAsync(w.err, 0, sizeof(int), st));
    int s = PMG_OK;
    const bool unit_res = ball_erode[0] >= 0.0;
    const float unit[3] = {1.0f, 1.0f, 1.0f};
    const float *r = unit_res ? unit : res;
    // radii that may share: their reach lies inside their own extension
    std::vector<char> shared((size_t)n_radii, 0);
    int n_shared = 0;
    for (int k = 0; k < n_radii; k++) {
        bool ok = (ball_erode[k] >= 0.0) == unit_res;
        const double reach = unit_res ? std::sqrt(ball_erode[k]) : radii[k];
        for (int d = 0; d < 3 && ok; d++)
            if (bc[2 * d] == PMG_BC_PERIODIC)
                ok = reach <= (double)ext[6 * (size_t)k + 2 * d] * r[d] &&
                     reach <= (double)ext[6 * (size_t)k + 2 * d + 1] * r[d];
        shared[(size_t)k] = ok;
        n_shared += ok;
    }
    float *D = nullptr;
    void *mem = nullptr;
    ExtRows XR{};
    if (n_shared > 1) {
        const size_t xb = morph_scratch_bytes(shape, bc, big);
        long long nx = 1;
        for (int d = 0; d < 3; d++)
            nx *= shape[d] + (bc[2 * d] == PMG_BC_PERIODIC ? big[2 * d] + big[2 * d + 1] : 0);
        const size_t tb = ((size_t)n_radii * 8 + 255) & ~(size_t)255;
        bool fits = nx < INT_MAX;
        for (int d = 0; d < 3; d++)
            fits = fits && shape[d] + big[2 * d] + big[2 * d + 1] <= PMG_MAX_LINE;
        const int got = fits ? scratch_alloc(&mem, xb + 256 + tb, st) : PMG_OK;
        if (got != PMG_OK) {
            // no room for the field: every radius by itself
            mem = nullptr;
            s = no_room(got) ? PMG_OK : got;
        } else if (fits) {
            uint8_t *E = (uint8_t *)mem;
            float *A = (float *)((char *)mem + (((size_t)nx + 255) & ~(size_t)255));
            D = A + nx;
            int64_t X[3], lo[3];
            const int ran = erosion_edt_ext_run(pm_img, D, shape, bc, pad, big, res, unit_res, E, A, X, lo, st);
            if (ran != PMG_OK) {
                D = nullptr; // (no room for its scratch)
                s = no_room(ran) ? PMG_OK : ran;
            }
            XR = ExtRows{X[1], X[2], lo[0], lo[1], lo[2]};
            const pmg_axis_cfg plain = {0, 0, 0, 0, 1, 0, 0, 0};
            bool exact = r[0] == r[1] && r[1] == r[2];
            for (int d = 0; d < 3 && exact; d++)
                exact = exact_path_ok(r[d], plain, (int)X[d]);
            if (D && !exact) {
                // the thresholds that may share (at: whose they are)
                std::vector<int> at((size_t)n_radii);
                auto of = [&](int k) { return (float)(unit_res ? ball_erode[k] : radii[k] * radii[k]); };
                for (int k = 0; k < n_radii; k++) {
                    at[(size_t)k] = k;
                    shared[(size_t)k] = shared[(size_t)k] && of(k) == of(k);
                }
                at.erase(std::remove_if(at.begin(), at.end(), [&](int k) { return !shared[(size_t)k]; }), at.end());
                const int m = (int)at.size();
                std::vector<float> thr((size_t)m);
                for (int k = 0; k < m; k++)
                    thr[(size_t)k] = of(at[(size_t)k]);
                float top = 0.0f;
                for (float t : thr)
                    top = t > top ? t : top;
                top = 2.0f * top + 4.0f * std::max(r[1] * r[1], r[2] * r[2]);
                float *dthr = (float *)((char *)mem + ((xb + 255) & ~(size_t)255));
                int *dflag = (int *)(dthr + n_radii);
                std::vector<int> flag((size_t)n_radii, 0);
                if (m > 0)
                    s = cudaMemcpyAsync(dthr, thr.data(), sizeof(float) * (size_t)m, cudaMemcpyHostToDevice, st) ==
                                    cudaSuccess &&
                                cudaMemsetAsync(dflag, 0, sizeof(int) * (size_t)m, st) == cudaSuccess
                            ? PMG_OK
                            : PMG_ECUDA;
                if (s == PMG_OK && m > 0) {
                    const int ps__ = prof_begin("k_near_thresholds", st);
                    k_near_thresholds<<<grid_for(shape[0] * shape[1] * 32, 256, 152LL * 32), 256, 0, st>>>(
                        D, shape[0], shape[1], shape[2], XR, dthr, m, top, r[1] * r[1], (float)X[1],
                        r[2] * r[2], (float)X[2], dflag);
                    prof_end(ps__, (double)n * 4, st);
                    s = cudaGetLastError() == cudaSuccess &&
                                cudaMemcpyAsync(flag.data(), dflag, sizeof(int) * (size_t)m, cudaMemcpyDeviceToHost,
                                                st) == cudaSuccess &&
                                cudaStreamSynchronize(st) == cudaSuccess
                            ? PMG_OK
                            : PMG_ECUDA;
                }
                for (int k = 0; k < m; k++)
                    if (flag[(size_t)k])
                        shared[(size_t)at[(size_t)k]] = 0;
            }
        }
    }
    uint8_t *todo = nullptr; // the pore voxels that no opening has covered yet
    if (s == PMG_OK)
        s = scratch_alloc((void **)&todo, (size_t)n, st);
    if (s == PMG_OK) {
        k_pore_mask<<<grid_for(n, 256, 152LL * 32), 256, 0, st>>>(pm_img, todo, n);
        s = cudaGetLastError() == cudaSuccess ? PMG_OK : PMG_ECUDA;
    }
    uint8_t *E;
    float *A, *B;
    for (int k = 0; k < n_radii && s == PMG_OK; k++) {
        const int32_t *e = ext.data() + 6 * (size_t)k;
        morph_split(w, shape, bc, e, E, A, B);
        uint8_t *cur = w.t1;
        if (D && shared[(size_t)k]) {
            ErodeThr T;
            T.lim = within_limit(radii[k], cmp64[k], ball_erode[k]);
            for (int q = 0; q < 6; q++)
                T.wall[q] = bc[q] == PMG_BC_WALL;
            const int ps__ = prof_begin("k_erode_from_edt", st);
            k_erode_from_edt<<<grid_for(shape[0] * shape[1] * 32, 256, 152LL * 64), 256, 0, st>>>(
                D, w.t1, shape[0], shape[1], shape[2], T, XR);
            prof_end(ps__, (double)n * 5, st);
            s = cudaGetLastError() == cudaSuccess ? PMG_OK : PMG_ECUDA;
        } else {
            s = morph_run(pm_img, w.t1, shape, bc, pad, e, res, radii[k], cmp64[k], 0, E, A, B, st, ball_erode[k]);
        }
        if (s == PMG_OK && inlet) {
            s = select_run_binary(w.t1, w.t2, 1, shape, bc, pad, Bx.inlet, nullptr, PMG_SEL_INLET, -1, w.P, w.M, w.mark,
                                  w.err, st, w.cnt);
            cur = w.t2;
        }
        // (the dilation of nothing is nothing)
        if (s == PMG_OK)
            s = morph_run(cur, w.t3, shape, bc, pad, e, res, radii[k], cmp64[k], 1, E, A, B, st, ball_dilate[k]);
        if (s == PMG_OK) {
            const int ps__ = prof_begin("k_first_cover", st);
            k_first_cover<<<grid_for(n / 16 + 1, 256, 152LL * 16), 256, 0, st>>>(w.t3, todo, out, radii[k], n);
            prof_end(ps__, (double)n * 2, st);
            s = cudaGetLastError() == cudaSuccess ? PMG_OK : PMG_ECUDA;
        }
    }
    if (s == PMG_OK && inlet)
        s = check_err(w.err, st);
    scratch_free(todo, st);
    scratch_free(mem, st);
    const int s2 = scratch_free(w.base, st);
    return s != PMG_OK ? s : s2;
}

extern "C" int pmg_drainage_ext(const uint8_t *pm_img, uint8_t *mp_img, const int64_t shape[3],
                                const int32_t bc[6], const int32_t pad[6], const int32_t rpad[6],
                                const int64_t own_box[6], const int64_t inlet_box[6],
                                const int64_t outlet_box[6], const float res[3], int32_t n_radii,
                                const double *radii, const int32_t *active, const int32_t *ratios,
                                const double *ball_erode, const double *ball_dilate, int64_t *counts,
                                const double *radii_dilate, const int32_t *ratios_dilate, void *stream)
{
    if (!radii_dilate)
        radii_dilate = radii;
    if (!ratios_dilate)
        ratios_dilate = ratios;
    PMG_TRY(check_common(shape, bc, pad));
    if (!pm_img || !mp_img || !rpad || !own_box || !res || !counts || n_radii < 0 ||
        (n_radii > 0 && (!radii || !active || !ratios))) {
        set_error("pmg_drainage: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_box6(shape, own_box));
    for (int q = 0; q < 6; q++)
        if (rpad[q] < 0) {
            set_error("pmg_drainage: negative reservoir pad");
            return PMG_EINVAL;
        }
    cudaStream_t st = as_stream(stream);
    const long long n = shape[0] * shape[1] * shape[2];
    Boxes Bx{};
    for (int q = 0; q < 6; q++) {
        Bx.own[q] = own_box[q];
        Bx.inlet[q] = inlet_box ? inlet_box[q] : -1;
        Bx.outlet[q] = outlet_box ? outlet_box[q] : -1;
        Bx.rpad[q] = rpad[q];
    }
    size_t mb = 0;
    for (int k = 0; k < n_radii; k++) {
        int32_t ext[6];
        ext_of(bc, pad, ratios + 3 * k, ext);
        size_t b = morph_scratch_bytes(shape, bc, ext);
        if (b > mb)
            mb = b;
        ext_of(bc, pad, ratios_dilate + 3 * k, ext);
        b = morph_scratch_bytes(shape, bc, ext);
        if (b > mb)
            mb = b;
    }
    Work w{};
    PMG_TRY(work_alloc(w, shape, mb, st));
    PMG_CUDA(cudaMemsetAsync(w.err, 0, sizeof(int), st));
    uint8_t *morph = nullptr;
    unsigned long long *d_counts = nullptr;
    // Without periodic axes the erosion's extended image is the same for every
    // radius (no wrap extension), so its EDT is computed once and thresholded
    // per radius -- the same values the per-radius EDT would produce.
    const bool reuse_erosion = bc[0] != PMG_BC_PERIODIC && bc[2] != PMG_BC_PERIODIC && bc[4] != PMG_BC_PERIODIC;
    float *De = nullptr;
    int unit_res = -1;
    for (int k = 0; k < n_radii; k++)
        if (active[k]) {
            unit_res = (ball_erode && ball_erode[k] >= 0.0) ? 1 : 0;
            break;
        }
    int s = PMG_OK;
    // Isotropic power-of-two voxels: the erosion EDT is kept as a capped
    // integer volume (uint16, values above the largest erosion bound clamp)
    // and each radius's erosion "E > T" is read off it inside the inlet
    // selection -- no eroded image is written.
    uint16_t *KC = nullptr;
    int Tcap = 0;
    std::vector<int> Te((size_t)n_radii, -1);
    if (reuse_erosion && unit_res >= 0) {
        const float unit[3] = {1.0f, 1.0f, 1.0f};
        const float *r = unit_res ? unit : res;
        const pmg_axis_cfg plain = {0, 0, 0, 0, 1, 0, 0, 0};
        bool ok = r[0] == r[1] && r[1] == r[2];
        for (int d = 0; d < 3 && ok; d++)
            ok = exact_path_ok(r[d], plain, (int)shape[d]);
        Tcap = 0;
        for (int k = 0; k < n_radii && ok; k++) {
            if (!active[k])
                continue;
            MorphEpi me{};
            me.lim = within_limit(radii[k], 1, ball_erode ? ball_erode[k] : -1.0);
            Te[(size_t)k] = morph_threshold(me, r[0] * r[0], kCapMaxT + 1);
            ok = Te[(size_t)k] >= 0 && Te[(size_t)k] <= kCapMaxT;
            Tcap = Te[(size_t)k] > Tcap ? Te[(size_t)k] : Tcap;
        }
        if (ok) {
            s = scratch_alloc((void **)&KC, (size_t)n * sizeof(uint16_t), st);
            int nonbinary = 0;
            if (s == PMG_OK) {
                uint8_t *E;
                float *A, *B;
                const int32_t zero_ext[6] = {0, 0, 0, 0, 0, 0};
                morph_split(w, shape, bc, zero_ext, E, A, B);
                s = erosion_cap_run(pm_img, KC, shape, bc, pad, Tcap, (uint16_t *)A, (uint16_t *)B,
                                    (int *)((char *)w.err + 128), &nonbinary, st);
            }
            if (s == PMG_OK && nonbinary) {
                s = scratch_free(KC, st);
                KC = nullptr;
            }
        }
    }
    if (s == PMG_OK && !KC && reuse_erosion && unit_res >= 0) {
        s = scratch_alloc((void **)&De, (size_t)n * sizeof(float), st);
        if (s == PMG_OK) {
            uint8_t *E;
            float *A, *B;
            const int32_t zero_ext[6] = {0, 0, 0, 0, 0, 0};
            morph_split(w, shape, bc, zero_ext, E, A, B);
            s = erosion_edt_run(pm_img, De, shape, bc, pad, res, unit_res, E, A, st);
        }
    }
    // The non-wetting phase only grows along the curve, and so does the eroded
    // pore space when the thresholds of the active radii never rise: both
    // selections keep their block union-find from one radius to the next.
    GrowSel g_er, g_nw;
    bool grow_er = KC != nullptr;
    {
        int last = INT_MAX;
        for (int k = 0; k < n_radii && grow_er; k++)
            if (active[k]) {
                grow_er = Te[(size_t)k] <= last;
                last = Te[(size_t)k];
            }
    }
    // the limits of the float distances (De) likewise
    std::vector<float> fthr;
    std::vector<uint8_t> fstep;
    if (De && n_radii <= 254) {
        bool ok = true;
        for (int k = 0; k < n_radii && ok; k++)
            if (active[k]) {
                const float t = within_limit(radii[k], 1, ball_erode ? ball_erode[k] : -1.0);
                ok = t == t && (fthr.empty() || t <= fthr.back());
                fthr.push_back(t);
                fstep.push_back((uint8_t)k);
            }
        grow_er = ok && !fthr.empty();
    }
    // the growing eroded space as one byte per voxel: the radius index at
    // which the voxel enters (the capped distances are not needed after it)
    uint8_t *Sv = nullptr;
    unsigned walls = 0;
    for (int q = 0; q < 6; q++)
        walls |= (bc[q] == PMG_BC_WALL ? 1u : 0u) << q;
    if (s == PMG_OK && grow_er && De) {
        const size_t m = fthr.size(), at = ((size_t)n + 255) & ~(size_t)255;
        s = scratch_alloc((void **)&Sv, at + m * (sizeof(float) + 1), st);
        float *dthr = (float *)(Sv + at);
        uint8_t *dstep = (uint8_t *)(dthr + m);
        // (a copy from pageable memory has read its source when it returns)
        if (s == PMG_OK && (cudaMemcpyAsync(dthr, fthr.data(), m * sizeof(float), cudaMemcpyHostToDevice, st) !=
                                cudaSuccess ||
                            cudaMemcpyAsync(dstep, fstep.data(), m, cudaMemcpyHostToDevice, st) != cudaSuccess))
            s = PMG_ECUDA;
        if (s == PMG_OK) {
            const int ps__ = prof_begin("k_step_volume", st);
            k_step_volume_f32<<<grid_for(shape[0] * shape[1] * 32, 256, 152LL * 64), 256, 0, st>>>(
                De, Sv, dthr, dstep, (int)m, shape[0], shape[1], shape[2], walls);
            prof_end(ps__, (double)n * 5, st);
            s = cudaGetLastError() == cudaSuccess ? PMG_OK : PMG_ECUDA;
        }
        if (s == PMG_OK) {
            s = scratch_free(De, st);
            De = nullptr;
        }
    }
    if (s == PMG_OK && grow_er && KC && n_radii <= 254) {
        std::vector<uint8_t> tab((size_t)Tcap + 2, 255);
        for (int v = 0; v <= Tcap + 1; v++)
            for (int k = 0; k < n_radii; k++)
                if (active[k] && Te[(size_t)k] < v) {
                    tab[(size_t)v] = (uint8_t)k;
                    break;
                }
        uint8_t *dtab = nullptr;
        s = scratch_alloc((void **)&Sv, (size_t)n + 256 + tab.size(), st);
        if (s == PMG_OK) {
            dtab = Sv + (((size_t)n + 255) & ~(size_t)255);
            s = cudaMemcpyAsync(dtab, tab.data(), tab.size(), cudaMemcpyHostToDevice, st) == cudaSuccess
                    ? PMG_OK
                    : PMG_ECUDA;
        }
        if (s == PMG_OK) {
            const int ps__ = prof_begin("k_step_volume", st);
            k_step_volume<<<grid_for(shape[0] * shape[1] * 32, 256, 152LL * 64), 256, 0, st>>>(
                KC, Sv, dtab, Tcap + 1, shape[0], shape[1], shape[2], walls);
            prof_end(ps__, (double)n * 3, st);
            // (a copy from pageable memory has read the table when it returns)
            s = cudaGetLastError() == cudaSuccess ? PMG_OK : PMG_ECUDA;
        }
        if (s == PMG_OK) {
            s = scratch_free(KC, st);
            KC = nullptr;
        }
    }
    void *grow_mem = nullptr;
    const size_t gb = grow_sel_bytes(shape), sb = shrink_sel_bytes(shape);
    if (s == PMG_OK)
        s = scratch_alloc(&grow_mem, gb * (grow_er ? 2 : 1) + sb, st);
    ShrinkSel g_w;
    if (s == PMG_OK)
        shrink_sel_init(g_w, (char *)grow_mem + gb * (grow_er ? 2 : 1), shape);
    if (s == PMG_OK) {
        grow_sel_init(g_nw, grow_mem, shape);
        if (grow_er)
            grow_sel_init(g_er, (char *)grow_mem + gb, shape);
    }
    // the blocks of the eroded space that grow at each radius, listed once
    void *lists_mem = nullptr;
    if (s == PMG_OK && Sv)
        s = step_lists_build(g_er, Sv, shape, n_radii, &lists_mem, st);
    // the dilation as bytes (paths that write them) and as row words
    unsigned *drows = nullptr;
    if (s == PMG_OK)
        s = scratch_alloc((void **)&morph, (((size_t)n + 255) & ~(size_t)255) + rows_bytes(shape), st);
    if (s == PMG_OK)
        drows = (unsigned *)(morph + (((size_t)n + 255) & ~(size_t)255));
    if (s == PMG_OK)
        s = scratch_alloc((void **)&d_counts, sizeof(unsigned long long) * (size_t)(n_radii + 1), st);
    if (s == PMG_OK)
        s = cudaMemsetAsync(d_counts, 0, sizeof(unsigned long long) * (size_t)(n_radii + 1), st) == cudaSuccess
                ? PMG_OK
                : PMG_ECUDA;
    // count(mp == 1) for the first radius; the update kernel keeps it current
    const int64_t whole[6] = {0, shape[0], 0, shape[1], 0, shape[2]};
    if (s == PMG_OK)
        s = cudaMemsetAsync(w.cnt + 1, 0, sizeof(unsigned long long), st) == cudaSuccess ? PMG_OK : PMG_ECUDA;
    if (s == PMG_OK)
        s = count_eq_async(mp_img, shape, whole, 1, w.cnt + 1, st);
    // After the first update (which refills the reservoir slabs), a radius can
    // change only voxels within the dilation's x range: the update visits that
    // range alone and counts changes (w.cnt[8], w.cnt[9]), the saturation count
    // being a running total (w.cnt[10]).
    int *orange = (int *)(w.cnt + 5);
    DrainCounts C{w.cnt + 8, w.cnt + 9, w.cnt + 10, w.cnt + 1, nullptr, w.cnt, (int *)(w.cnt + 4),
                  (unsigned *)(w.cnt + 11)};
    if (s == PMG_OK)
        s = cudaMemsetAsync(w.cnt, 0, sizeof(unsigned long long), st) == cudaSuccess &&
                    cudaMemsetAsync(w.cnt + 4, 0, 8 * sizeof(unsigned long long), st) == cudaSuccess
                ? PMG_OK
                : PMG_ECUDA;
    // The wetting phase's union-find depends on the last update alone: it runs on
    // a stream of its own beside the selection and the dilation, whose kernels
    // leave much of the chip waiting on dependent loads.  The eroded space does
    // not depend on the phases at all: a third stream prepares the next radius's
    // while this one's selection is dilated.
    Fork fork, eroded;
    if (s == PMG_OK)
        s = fork.open();
    if (s == PMG_OK && grow_er)
        s = eroded.open();
    auto next_eroded = [&](int k) -> int {
        while (k < n_radii && !active[k])
            k++;
        if (!grow_er || k == n_radii)
            return PMG_OK;
        const int s1 = grow_marks_eroded(g_er, Sv, k, KC, Te[(size_t)k], shape, bc, pad, Bx.inlet, w.err, eroded.side);
        const int s2 = eroded.end();
        return s1 != PMG_OK ? s1 : s2;
    };
    if (s == PMG_OK && grow_er)
        s = eroded.begin(st);
    if (s == PMG_OK)
        s = next_eroded(0);
    bool full_done = false;
    for (int k = 0; k < n_radii && s == PMG_OK; k++) {
        C.sat = d_counts + k;
        if (!active[k] && full_done) {
            // no dilation: nothing changes, the totals stand
            s = drain_same(C, st);
            continue;
        }
        // wetting phase connected to the outlet (its union-find and stamps
        // only; tiles the last update left alone keep their tile-local parents)
        s = fork.begin(st);
        if (s == PMG_OK) {
            s = shrink_marks_binary(g_w, mp_img, 2, shape, bc, pad, Bx.outlet, w.err, fork.side);
            const int s1 = fork.end();
            s = s == PMG_OK ? s1 : s;
        }
        if (active[k] && s == PMG_OK) {
            int32_t ext[6], ext_d[6];
            ext_of(bc, pad, ratios + 3 * k, ext);
            ext_of(bc, pad, ratios_dilate + 3 * k, ext_d);
            // the probe radii are numpy float64: compare in float64
            s = porosimetry_run(pm_img, morph, shape, bc, pad, ext, ext_d, res, radii[k], 1, radii_dilate[k], 1, 1,
                                mp_img,
                                Bx, w, st, ball_erode ? ball_erode[k] : -1.0, ball_dilate ? ball_dilate[k] : -1.0,
                                De, KC, Te[(size_t)k], true, grow_er ? &g_er : nullptr, &g_nw, orange, drows,
                                grow_er ? &eroded : nullptr);
            if (s == PMG_OK)
                s = next_eroded(k + 1);
        }
        {
            // (also after an error: the scratch below is freed in st's order)
            const int s1 = fork.join(st);
            s = s == PMG_OK ? s1 : s;
        }
        if (s != PMG_OK)
            break;
        // the update on row words, which also brings the non-wetting phase's
        // growing selection and the wetting phase's masks and tile flags up to date
        GrowSel *gn = g_nw.built ? &g_nw : nullptr;
        s = drain_update_rows(mp_img, active[k] ? drows : nullptr, shape, g_w, Bx, gn, C, w.err, st,
                              active[k] ? orange : nullptr, !full_done);
        if (s != PMG_OK)
            break;
        full_done = true;
        if (gn)
            gn->pending = true;
    }
    {
        // (scratch is freed in st's order)
        const int s1 = eroded.join(st);
        s = s == PMG_OK ? s1 : s;
    }
    // union-find iteration caps are checked once per curve: the status word
    // is only ever set, never cleared, during the sweep
    if (s == PMG_OK)
        s = check_err(w.err, st);
    if (s == PMG_OK && n_radii > 0) {
        std::vector<unsigned long long> h((size_t)n_radii);
        PMG_CUDA(cudaMemcpyAsync(h.data(), d_counts, sizeof(unsigned long long) * (size_t)n_radii,
                                 cudaMemcpyDeviceToHost, st));
        PMG_CUDA(cudaStreamSynchronize(st));
        for (int k = 0; k < n_radii; k++)
            counts[k] = (int64_t)h[(size_t)k];
    }
    scratch_free(lists_mem, st);
    scratch_free(grow_mem, st);
    scratch_free(Sv, st);
    scratch_free(De, st);
    scratch_free(KC, st);
    scratch_free(morph, st);
    scratch_free(d_counts, st);
    int s2 = scratch_free(w.base, st);
    return s != PMG_OK ? s : s2;
}

extern "C" int pmg_drainage(const uint8_t *pm_img, uint8_t *mp_img, const int64_t shape[3],
                            const int32_t bc[6], const int32_t pad[6], const int32_t rpad[6],
                            const int64_t own_box[6], const int64_t inlet_box[6],
                            const int64_t outlet_box[6], const float res[3], int32_t n_radii,
                            const double *radii, const int32_t *active, const int32_t *ratios,
                            const double *ball_erode, const double *ball_dilate, int64_t *counts,
                            void *stream)
{
    return pmg_drainage_ext(pm_img, mp_img, shape, bc, pad, rpad, own_box, inlet_box, outlet_box, res, n_radii,
                            radii, active, ratios, ball_erode, ball_dilate, counts, nullptr, nullptr, stream);
}
