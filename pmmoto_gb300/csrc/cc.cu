// Connected components on GB300 (sm_103a).
//
// Reference: pmmoto.filters.connected_components (src/pmmoto/filters/
// connected_components.py:32-392) -- labelling by the third-party cc3d
// (26-connectivity, each nonzero value separately, background 0), periodic
// seam merge (connect_subdomain_boundaries :65-101 with core/voxels.py:
// 167-397 and core/_voxels.pyx:335-383, 548-579), inlet/outlet selection
// (:144-392, voxels.py:400-454).
//
// Device algorithm: lock-free union-find over voxel indices where a union
// always links the larger root under the smaller, so a component's final root
// is its smallest voxel index -- its first voxel in C-order raster scan.
// Numbering components by the rank of their root therefore numbers them in
// order of first appearance, the order cc3d issues labels.  Elements of a row
// that touch form runs, and one union is made per pair of touching runs of
// neighbouring rows, which removes most redundant unions.  Periodic seams are
// united voxel-with-twin (the voxel its halo copies), which is what the
// reference's pair matching does.
//
// Every data-dependent loop carries an iteration cap; hitting it sets a
// device status word and the entry point returns PMG_EITER.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <type_traits>
#include <array>
#include <unordered_map>
#include <unordered_set>
#include <vector>

#include "pmg_common.cuh"
#include "pmg_internal.cuh"
#include "uf.cuh"

namespace pmg {

struct Vol3 {
    long long s0, s1, s2;
};

// ---- tiled labelling ------------------------------------------------------
// Tiles of 4 x 8 x 32 elements (C order, the last axis contiguous; voxels here,
// 2x2x2 blocks below), 32 rows of 32, one warp per row in the first phase.
// Phase 1 unites the parts of a tile with a shared-memory union-find whose
// roots are the smallest local index -- which is also the smallest global
// index of that part of the component, because C order inside a box follows
// the global C order.  Phase 2 unites across tile borders through the global
// parents.  Both work on runs: touching neighbours of a row share the run's
// first element (the head) as parent, and of the touching pairs of two
// neighbouring rows one per pair of runs is united.
constexpr int kT0 = 4, kT1 = 8, kT2 = 32, kTile = kT0 * kT1 * kT2;

__device__ __forceinline__ int sfind(const int *L, int x)
{
    int p = L[x];
    int it = 0;
    while (p != x && it++ < kTile) {
        x = p;
        p = L[x];
    }
    return x;
}

// root search with path halving (same argument as find_root_halve)
__device__ __forceinline__ int sfind_halve(int *L, int x)
{
    int p = L[x];
    int it = 0;
    while (p != x && it++ < kTile) {
        const int g = L[p];
        if (g == p)
            return p;
        L[x] = g;
        x = g;
        p = L[x];
    }
    return x;
}

__device__ __forceinline__ void sunite(int *L, int a, int b)
{
    for (int it = 0; it < 4 * kTile; it++) {
        a = sfind_halve(L, a);
        b = sfind_halve(L, b);
        if (a == b)
            return;
        if (a < b) {
            const int old = atomicMin(L + b, a);
            if (old == b)
                return;
            b = old;
        } else {
            const int old = atomicMin(L + a, b);
            if (old == a)
                return;
            a = old;
        }
    }
}

// first element of the run of element c; cz: elements joined to the one before
__device__ __forceinline__ int run_head(unsigned cz, int c) { return 31 - __clz(~cz & (0xffffffffu >> (31 - c))); }

// neighbouring row q = 0..3: (-1, 0), (-1, -1), (-1, 1), (0, -1)
__device__ __forceinline__ int row_d0(int q) { return q < 3 ? -1 : 0; }
__device__ __forceinline__ int row_d1(int q) { return q == 0 ? 0 : q == 2 ? 1 : -1; }

// Of the touching pairs of a row's elements with the ones before (em), beside
// (e0) and after (ep) them in a neighbouring row, one per pair of runs: cz, bz
// are the runs of the row and of its neighbour.  A straight pair is dropped
// when the element before makes one between the same two runs, a slanted one
// when a straight one does.
__device__ __forceinline__ void row_reduce(unsigned cz, unsigned bz, unsigned &em, unsigned &e0, unsigned &ep)
{
    const unsigned s0 = e0;
    e0 &= ~(cz & (s0 << 1) & bz);
    em &= ~((s0 & bz) | (cz & (s0 << 1)));
    ep &= ~((s0 & (bz >> 1)) | ((cz >> 1) & (s0 >> 1)));
}

// Row pairs across a tile's borders: the a = 0 plane's rows with the three rows
// above, then the rows before b = 0, then the slanted ones of the other planes.
constexpr int kCrossPairs = kT1 * 3 + kT0 + (kT0 - 1) * 2;

__device__ __forceinline__ void cross_pair(int i, int &a, int &b, int &q)
{
    if (i < kT1 * 3) {
        a = 0;
        b = i / 3;
        q = i % 3;
    } else if (i < kT1 * 3 + kT0) {
        a = i - kT1 * 3;
        b = 0;
        q = 3;
    } else {
        const int k = i - kT1 * 3 - kT0;
        a = 1 + k / 2;
        b = (k & 1) * (kT1 - 1);
        q = 1 + (k & 1);
    }
}

// Unions across a tile's borders.  Phase 1 left every element's tile-local root
// in P, so two touching elements stand for a pair of tile-local components: a
// shared-memory set of the pairs seen keeps all but the first of each pair
// from the global union-find (a tile has a few components, and hundreds of
// touching pairs).  Pairs are listed and then taken by all threads of the
// block: a thread's own would run one after the other, each a chain of
// dependent loads.
constexpr int kPairSlots = 256, kPairProbes = 8, kPairList = 768;

struct CrossSet {
    unsigned long long set[kPairSlots];
    int2 list[kPairList];
    int count;

    __device__ __forceinline__ void init()
    {
        for (int q = threadIdx.x; q < kPairSlots; q += blockDim.x)
            set[q] = ~0ull;
        if (threadIdx.x == 0)
            count = 0;
        __syncthreads();
    }
    // True when this pair has been seen in the block (its union is done by
    // another thread); a full set lets pairs through.
    __device__ __forceinline__ bool seen(int pa, int pb)
    {
        const unsigned long long key = ((unsigned long long)(unsigned)pa << 32) | (unsigned)pb;
        unsigned h = ((unsigned)pa * 2654435761u) ^ ((unsigned)pb * 2246822519u);
        h = (h ^ (h >> 15)) % kPairSlots;
        for (int i = 0; i < kPairProbes; i++) {
            const unsigned long long old = atomicCAS(set + h, ~0ull, key);
            if (old == ~0ull)
                return false;
            if (old == key)
                return true;
            h = (h + 1) % kPairSlots;
        }
        return false;
    }
    __device__ __forceinline__ void join(int *P, int x, int y, int *err)
    {
        const int px = ld(P + x), py = ld(P + y);
        if (px != py && !seen(px, py))
            unite(P, px, py, err);
    }
    __device__ __forceinline__ void add(int *P, int x, int y, int *err)
    {
        const int k = atomicAdd(&count, 1);
        if (k < kPairList)
            list[k] = make_int2(x, y);
        else
            join(P, x, y, err);
    }
    // after every add of the block
    __device__ __forceinline__ void finish(int *P, int *err)
    {
        __syncthreads();
        const int total = min(count, kPairList);
        for (int k = threadIdx.x; k < total; k += blockDim.x)
            join(P, list[k].x, list[k].y, err);
    }
};

// Grid of the tile kernels: tiles (x along the contiguous axis).
struct TileId {
    int ti, tj, tk, nt1, nt2;
    __device__ __forceinline__ TileId()
        : ti(blockIdx.z), tj(blockIdx.y), tk(blockIdx.x), nt1(gridDim.y), nt2(gridDim.x)
    {
    }
    __device__ __forceinline__ int index() const { return (ti * nt1 + tj) * nt2 + tk; }
};

// Phase 1 on voxels (equal nonzero neighbours touch).  A voxel equal to the one
// above it leaves its other earlier neighbours to that one: it is adjacent to
// all of them.  A warp takes four rows, whose loads overlap; the pairs of a row
// with one of its neighbouring rows are then united by one lane (lane 4 u + q:
// row u, neighbour q).
// A tile is a chain of dependent steps between barriers: with a thread per voxel
// (1024 of them, two tiles in flight on an SM) this took 244 us on 257 x 200 x 323
// voxels, now 174 us.
constexpr int kCcTileThreads = 256, kCcRows = kTile / kCcTileThreads;

template <typename T>
__global__ void __launch_bounds__(kCcTileThreads) k_cc_tile(const T *__restrict__ img, int *__restrict__ P, Vol3 V)
{
    __shared__ T sv[kTile];
    __shared__ int L[kTile];
    __shared__ unsigned s_cz[kT0 * kT1];
    const TileId D;
    const int w = threadIdx.x / kT2, lane = threadIdx.x % kT2, k = D.tk * kT2 + lane;
    T v[kCcRows];
    unsigned cz[kCcRows];
    long long g[kCcRows]; // -1: outside
#pragma unroll
    for (int u = 0; u < kCcRows; u++) {
        const int r = w * kCcRows + u, i = D.ti * kT0 + r / kT1, j = D.tj * kT1 + r % kT1;
        const bool inside = i < V.s0 && j < V.s1 && k < V.s2;
        g[u] = inside ? ((long long)i * V.s1 + j) * V.s2 + k : -1;
        v[u] = inside ? img[g[u]] : (T)0;
    }
#pragma unroll
    for (int u = 0; u < kCcRows; u++) {
        const int r = w * kCcRows + u;
        sv[r * kT2 + lane] = v[u];
        const T vp = __shfl_up_sync(0xffffffffu, v[u], 1);
        cz[u] = __ballot_sync(0xffffffffu, lane > 0 && v[u] != 0 && v[u] == vp);
        L[r * kT2 + lane] = v[u] != 0 ? r * kT2 + run_head(cz[u], lane) : -1;
        if (lane == 0)
            s_cz[r] = cz[u];
    }
    __syncthreads();
    unsigned em = 0, e0 = 0, ep = 0; // of this lane's pair of rows
#pragma unroll
    for (int u = 0; u < kCcRows; u++) {
        const int r = w * kCcRows + u, a = r / kT1, b = r % kT1;
        if (!__any_sync(0xffffffffu, v[u] != 0))
            continue;
        bool centre = false;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (a + row_d0(q) < 0 || b + row_d1(q) < 0 || b + row_d1(q) >= kT1)
                continue;
            const int rn = r + row_d0(q) * kT1 + row_d1(q);
            const T n0 = sv[rn * kT2 + lane], nm = __shfl_up_sync(0xffffffffu, n0, 1),
                    np = __shfl_down_sync(0xffffffffu, n0, 1);
            const bool on = v[u] != 0 && !centre;
            const unsigned E0 = __ballot_sync(0xffffffffu, on && n0 == v[u]),
                           Em = __ballot_sync(0xffffffffu, on && lane > 0 && nm == v[u]),
                           Ep = __ballot_sync(0xffffffffu, on && lane < 31 && np == v[u]);
            if (q == 0)
                centre = (E0 >> lane) & 1u;
            if (lane == 4 * u + q) {
                em = Em;
                e0 = E0;
                ep = Ep;
            }
        }
    }
    if (em | e0 | ep) {
        const int q = lane & 3, r = w * kCcRows + (lane >> 2), rn = r + row_d0(q) * kT1 + row_d1(q);
        const unsigned ca = s_cz[r], cb = s_cz[rn];
        row_reduce(ca, cb, em, e0, ep);
        while (em | e0 | ep) {
            const int dz = e0 ? 0 : em ? -1 : 1;
            const unsigned e = e0 ? e0 : em ? em : ep;
            const int c = __ffs(e) - 1;
            const unsigned bit = e & (0u - e);
            e0 &= ~(dz == 0 ? bit : 0u);
            em &= ~(dz < 0 ? bit : 0u);
            ep &= ~(dz > 0 ? bit : 0u);
            sunite(L, r * kT2 + run_head(ca, c), rn * kT2 + run_head(cb, c + dz));
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kCcRows; u++) {
        const int r = w * kCcRows + u, head = run_head(cz[u], lane);
        int root = -1;
        if (v[u] != 0 && head == lane)
            root = sfind(L, r * kT2 + lane);
        root = __shfl_sync(0xffffffffu, root, head);
        if (g[u] >= 0) {
            int out = -1;
            if (v[u] != 0) {
                const int ra = root / (kT1 * kT2), rb = (root / kT2) % kT1, rc = root % kT2;
                out = (int)(((long long)(D.ti * kT0 + ra) * V.s1 + D.tj * kT1 + rb) * V.s2 + D.tk * kT2 + rc);
            }
            P[g[u]] = out;
        }
    }
}

// Phase 2 on voxels: a warp per row pair in different tiles, then a thread per
// row end (slanted neighbours, and straight ones at the low end, lie in the
// tiles beside).
constexpr int kCcCrossThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kCcCrossThreads) k_cc_cross(const T *__restrict__ img, int *P, Vol3 V, int *err)
{
    __shared__ CrossSet S;
    const TileId D;
    S.init();
    // volumes are below 2^31 voxels, so 32-bit index arithmetic suffices
    const int S0 = (int)V.s0, S1 = (int)V.s1, S2 = (int)V.s2;
    const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int pi = w; pi < kCrossPairs; pi += kCcCrossThreads / 32) {
        int a, b, q;
        cross_pair(pi, a, b, q);
        const int i = D.ti * kT0 + a, j = D.tj * kT1 + b, k = D.tk * kT2 + lane, ni = i + row_d0(q),
                  nj = j + row_d1(q);
        if (i >= S0 || j >= S1 || ni < 0 || nj < 0 || nj >= S1)
            continue;
        const int x = (i * S1 + j) * S2 + k, y = (ni * S1 + nj) * S2 + k;
        const T v = k < S2 ? img[x] : (T)0, n0 = k < S2 ? img[y] : (T)0;
        const T vp = __shfl_up_sync(0xffffffffu, v, 1);
        T nm = __shfl_up_sync(0xffffffffu, n0, 1), np = __shfl_down_sync(0xffffffffu, n0, 1);
        const unsigned cz = __ballot_sync(0xffffffffu, lane > 0 && v != 0 && v == vp),
                       bz = __ballot_sync(0xffffffffu, lane > 0 && n0 != 0 && n0 == nm);
        if (lane == 0)
            nm = k > 0 ? img[y - 1] : (T)0;
        if (lane == 31)
            np = k + 1 < S2 ? img[y + 1] : (T)0;
        unsigned E0 = __ballot_sync(0xffffffffu, v != 0 && n0 == v), Em = __ballot_sync(0xffffffffu, v != 0 && nm == v),
                 Ep = __ballot_sync(0xffffffffu, v != 0 && np == v);
        row_reduce(cz, bz, Em, E0, Ep);
        if ((E0 >> lane) & 1u)
            S.add(P, x, y, err);
        if ((Em >> lane) & 1u)
            S.add(P, x, y - 1, err);
        if ((Ep >> lane) & 1u)
            S.add(P, x, y + 1, err);
    }
    if (threadIdx.x < kT0 * kT1 * 2) {
        const int r = threadIdx.x >> 1, a = r / kT1, b = r % kT1;
        const bool low = !(threadIdx.x & 1);
        const int dz = low ? -1 : 1;
        const int i = D.ti * kT0 + a, j = D.tj * kT1 + b, k = D.tk * kT2 + (low ? 0 : kT2 - 1);
        if (i < S0 && j < S1 && k < S2 && k + dz >= 0 && k + dz < S2) {
            const int x = (i * S1 + j) * S2 + k;
            const T v = img[x];
            if (v != 0) {
                if (low && img[x - 1] == v)
                    S.add(P, x, x - 1, err);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (a + row_d0(q) < 0 || b + row_d1(q) < 0 || b + row_d1(q) >= kT1 || j + row_d1(q) >= S1)
                        continue; // (a row pair's, or outside)
                    const int y = x + (row_d0(q) * S1 + row_d1(q)) * S2 + dz;
                    if (img[y] == v)
                        S.add(P, x, y, err);
                }
            }
        }
    }
    S.finish(P, err);
}

// Seam twins of the voxel labelling (see Twins).
template <typename T>
__global__ void k_cc_twins(const T *__restrict__ img, int *P, Twins W, int *err)
{
    const long long n = W.s0 * W.s1 * W.s2;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        long long c[3];
        c[2] = idx % W.s2;
        long long r = idx / W.s2;
        c[1] = r % W.s1;
        c[0] = r / W.s1;
        bool halo = false;
        long long t[3];
        bool ok = true;
        for (int d = 0; d < 3; d++) {
            t[d] = c[d];
            const long long S = d == 0 ? W.s0 : d == 1 ? W.s1 : W.s2;
            const bool in_halo = c[d] < W.own_lo[d] || c[d] >= W.own_lo[d] + W.own_len[d];
            if (in_halo) {
                if (!W.periodic[d] || W.own_len[d] <= 0 || c[d] < 0 || c[d] >= S) {
                    ok = false;
                } else {
                    long long q = (c[d] - W.own_lo[d]) % W.own_len[d];
                    if (q < 0)
                        q += W.own_len[d];
                    t[d] = q + W.own_lo[d];
                    halo = true;
                }
            }
        }
        if (!halo || !ok || img[idx] == 0)
            continue;
        const long long tw = (t[0] * W.s1 + t[1]) * W.s2 + t[2];
        if (img[tw] != 0)
            unite(P, (int)idx, (int)tw, err);
    }
}

// Four voxels per thread: their chains of dependent loads overlap.
__global__ void __launch_bounds__(256) k_cc_flatten(int *P, long long n, int *err)
{
    constexpr int NB = 4;
    for (long long base = (long long)blockIdx.x * blockDim.x * NB; base < n;
         base += (long long)gridDim.x * blockDim.x * NB) {
        int p[NB], g[NB];
#pragma unroll
        for (int q = 0; q < NB; q++) {
            const long long i = base + q * blockDim.x + threadIdx.x;
            p[q] = i < n ? ld(P + i) : -1;
        }
#pragma unroll
        for (int q = 0; q < NB; q++)
            g[q] = p[q] >= 0 ? ld(P + p[q]) : -1;
#pragma unroll
        for (int q = 0; q < NB; q++)
            if (g[q] != p[q])
                P[base + q * blockDim.x + threadIdx.x] = find_root(P, g[q], err);
    }
}

// ---- numbering by root order -------------------------------------------
constexpr int kNumBlock = 512;
constexpr int kNumItems = 4; // voxels per thread in the numbering kernels
constexpr long long kNumTile = (long long)kNumBlock * kNumItems;

__global__ void k_root_count(const int *__restrict__ P, long long n, int *__restrict__ counts)
{
    typedef cub::BlockReduce<int, kNumBlock> BR;
    __shared__ typename BR::TempStorage tmp;
    const long long base = blockIdx.x * kNumTile;
    int c = 0;
#pragma unroll
    for (int q = 0; q < kNumItems; q++) {
        const long long i = base + (long long)threadIdx.x * kNumItems + q;
        if (i < n && P[i] == (int)i)
            c++;
    }
    const int tot = BR(tmp).Sum(c);
    if (threadIdx.x == 0)
        counts[blockIdx.x] = tot;
}

// R[i] = rank of root i among all roots (0-based); P is left unchanged.
__global__ void k_root_rank(const int *__restrict__ P, long long n, const int *__restrict__ offs,
                            int *__restrict__ R)
{
    typedef cub::BlockScan<int, kNumBlock> BS;
    __shared__ typename BS::TempStorage tmp;
    const long long base = blockIdx.x * kNumTile;
    int f[kNumItems];
#pragma unroll
    for (int q = 0; q < kNumItems; q++) {
        const long long i = base + (long long)threadIdx.x * kNumItems + q;
        f[q] = (i < n && P[i] == (int)i) ? 1 : 0;
    }
    int x[kNumItems];
    BS(tmp).ExclusiveSum(f, x);
#pragma unroll
    for (int q = 0; q < kNumItems; q++) {
        const long long i = base + (long long)threadIdx.x * kNumItems + q;
        if (f[q])
            R[i] = offs[blockIdx.x] + x[q];
    }
}

__global__ void k_label_out(const int *__restrict__ P, const int *__restrict__ R, long long n,
                            uint64_t *__restrict__ L)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const int p = P[i];
        L[i] = p < 0 ? 0ull : (uint64_t)R[p] + 1ull;
    }
}

// ---- seam pairs for the reference's periodic numbering --------------------

// keys[r] = label(own/neighbour voxel r) << 32 | label(twin), rows in the
// reference's order: own slab then neighbour slab of the feature, each
// flattened in C order, paired with the opposite feature's neighbour then own.
// Labels read from a label volume ...
struct LabImg {
    const uint64_t *L;
    Vol3 V;
    __device__ __forceinline__ uint64_t at(long long i, long long j, long long k) const
    {
        return L[(i * V.s1 + j) * V.s2 + k];
    }
};

// keys[row0 + r] = fkey | label << lbits | twin label (fkey = 0, lbits = 32
// for one feature alone), idx[row0 + r] = row0 + r.
template <class Src>
__global__ void k_seam_pairs(Src src, Box a0, Box a1, Box b0, Box b1, uint64_t fkey, int lbits, long long row0,
                             uint64_t *__restrict__ keys, uint32_t *__restrict__ idx)
{
    keys += row0;
    idx += row0;
    const long long n0 = a0.size(), n = n0 + a1.size();
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n;
         r += (long long)gridDim.x * blockDim.x) {
        const Box &A = r < n0 ? a0 : a1;
        const Box &B = r < n0 ? b0 : b1;
        const long long q = r < n0 ? r : r - n0;
        const long long wa = A.hi[2] - A.lo[2], ha = A.hi[1] - A.lo[1];
        const long long wb = B.hi[2] - B.lo[2], hb = B.hi[1] - B.lo[1];
        const long long ak = q % wa, aj = (q / wa) % ha, ai = q / (wa * ha);
        const long long bk = q % wb, bj = (q / wb) % hb, bi = q / (wb * hb);
        const uint64_t la = src.at(A.lo[0] + ai, A.lo[1] + aj, A.lo[2] + ak);
        const uint64_t lb = src.at(B.lo[0] + bi, B.lo[1] + bj, B.lo[2] + bk);
        keys[r] = fkey | (la << lbits) | lb;
        idx[r] = (uint32_t)(row0 + r);
    }
}

__global__ void k_head_flags(const uint64_t *__restrict__ k, long long n, uint8_t *__restrict__ f)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        f[i] = (i == 0 || k[i] != k[i - 1]) ? 1 : 0;
}

__global__ void k_apply_lut(uint64_t *L, long long n, const uint64_t *__restrict__ lut)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        L[i] = lut[L[i]];
}

__global__ void k_lut_flags(const uint64_t *__restrict__ bl, const uint64_t *__restrict__ bg, long long nbnd,
                            uint8_t *__restrict__ flag, uint64_t *__restrict__ lut)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nbnd;
         i += (long long)gridDim.x * blockDim.x) {
        flag[bl[i]] = 1;
        lut[bl[i]] = bg[i];
    }
}

__global__ void k_lut_nonflag(const uint8_t *__restrict__ flag, long long m, int *__restrict__ nf)
{
    for (long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x; l < m;
         l += (long long)gridDim.x * blockDim.x)
        nf[l] = (l > 0 && !flag[l]) ? 1 : 0;
}

__global__ void k_lut_fill(const uint8_t *__restrict__ flag, const int *__restrict__ rank, long long m,
                           uint64_t start, uint64_t *__restrict__ lut)
{
    for (long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x; l < m;
         l += (long long)gridDim.x * blockDim.x) {
        if (l == 0)
            lut[0] = 0;
        else if (!flag[l])
            lut[l] = start + (uint64_t)rank[l];
    }
}

// ---- inlet / outlet selection ---------------------------------------------
__global__ void k_mark_face(const int *__restrict__ P, Vol3 V, Box b, uint8_t *__restrict__ mark,
                            uint8_t bit)
{
    const long long n = b.size();
    const long long w = b.hi[2] - b.lo[2], h = b.hi[1] - b.lo[1];
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const long long k = q % w, j = (q / w) % h, i = q / (w * h);
        const long long idx = ((b.lo[0] + i) * V.s1 + b.lo[1] + j) * V.s2 + b.lo[2] + k;
        const int p = P[idx];
        if (p >= 0 && !(mark[p] & bit))
            atomicOr((unsigned int *)(mark + (p & ~3ll)), (unsigned int)bit << (8 * (p & 3)));
    }
}

template <typename TO>
__global__ void k_select(const uint8_t *__restrict__ img, const int *__restrict__ P,
                         const uint8_t *__restrict__ mark, long long n, int mode, int phase,
                         TO *__restrict__ out)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const uint8_t v = img[i];
        const int p = P[i];
        TO o = 0;
        if (v != 0 && p >= 0 && (phase < 0 || v == phase)) {
            const uint8_t m = mark[p];
            const bool in = m & 1, ou = m & 2;
            bool keep;
            if (mode == PMG_SEL_INLET)
                keep = in;
            else if (mode == PMG_SEL_OUTLET)
                keep = ou;
            else if (mode == PMG_SEL_BOTH)
                keep = in && ou;
            else
                keep = !(in || ou);
            if (keep)
                o = (TO)v;
        }
        out[i] = o;
    }
}

// ---------------------------------------------------------------------------
// Union-find of a volume into P (roots = smallest index); twins optional.
template <typename T>
static int uf_build(const T *img, int *P, const int64_t *shape, const int32_t *bc,
                    const int32_t *pad, bool twins, int *err, cudaStream_t st)
{
    const long long n = shape[0] * shape[1] * shape[2];
    Vol3 V{shape[0], shape[1], shape[2]};
    const int block = 256;
    const dim3 tiles((unsigned)((shape[2] + kT2 - 1) / kT2), (unsigned)((shape[1] + kT1 - 1) / kT1),
                     (unsigned)((shape[0] + kT0 - 1) / kT0));
    {
        const int ps__ = prof_begin("k_cc_tile", st);
        k_cc_tile<T><<<tiles, kCcTileThreads, 0, st>>>(img, P, V);
        prof_end(ps__, (double)n * (sizeof(T) + 4), st);
    }
    PMG_CHECK_LAUNCH();
    {
        const int ps__ = prof_begin("k_cc_cross", st);
        k_cc_cross<T><<<tiles, kCcCrossThreads, 0, st>>>(img, P, V, err);
        prof_end(ps__, 0.0, st);
    }
    PMG_CHECK_LAUNCH();
    if (twins && any_periodic(bc)) {
        {
            const int ps__ = prof_begin("k_cc_twins", st);
            k_cc_twins<T><<<grid_for(n, block, 152LL * 32), block, 0, st>>>(img, P,
                                                                         make_twins(shape, bc, pad), err);
            prof_end(ps__, 0.0, st);
        }
        PMG_CHECK_LAUNCH();
    }
    {
        const int ps__ = prof_begin("k_cc_flatten", st);
        k_cc_flatten<<<grid_for((n + 3) / 4, block, 152LL * 32), block, 0, st>>>(P, n, err);
        prof_end(ps__, (double)n * 8, st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

static int read_err(int *err, cudaStream_t st)
{
    int h = 0;
    PMG_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    PMG_CUDA(cudaStreamSynchronize(st));
    if (h == 3) {
        set_error("connected components: a growing-set selection lost voxels between steps");
        return PMG_EINVAL;
    }
    if (h != 0) {
        set_error("connected components: union-find iteration cap reached (code %d)", h);
        return PMG_EITER;
    }
    return PMG_OK;
}

// Feature slabs (src/pmmoto/core/features.py:76-139) of a single-rank
// padded subdomain; `kind` is the feature's boundary kind (boundary_order).
static void feature_slabs(const int f[3], int kind, const int64_t *shape, const int32_t *pad,
                          Box &own, Box &nb)
{
    bool padded = false;
    for (int d = 0; d < 6; d++)
        padded |= pad[d] != 0;
    for (int d = 0; d < 3; d++) {
        const long long L = shape[d], pb = pad[2 * d], pa = pad[2 * d + 1];
        if (f[d] == -1) {
            if (pb && kind != PMG_BC_WALL) {
                own.lo[d] = pb;
                own.hi[d] = 2 * pb;
            } else if (pb) {
                own.lo[d] = 1;
                own.hi[d] = 2;
            } else {
                own.lo[d] = 0;
                own.hi[d] = 1;
            }
            nb.lo[d] = 0;
            nb.hi[d] = padded ? (kind == PMG_BC_WALL ? 1 : pb) : 0;
        } else if (f[d] == 1) {
            if (pa && kind != PMG_BC_WALL) {
                own.lo[d] = L - 2 * pa;
                own.hi[d] = L - pa;
            } else if (pa) {
                own.lo[d] = L - 2;
                own.hi[d] = L - 1;
            } else {
                own.lo[d] = L - 1;
                own.hi[d] = L;
            }
            nb.lo[d] = padded ? (kind == PMG_BC_WALL ? L - 1 : L - pa) : 0;
            nb.hi[d] = padded ? L : 0;
        } else {
            own.lo[d] = pb;
            own.hi[d] = L - pa;
            nb.lo[d] = padded ? pb : 0;
            nb.hi[d] = padded ? L - pa : 0;
        }
    }
}

// Features in the reference's iteration order (faces, edges, corners;
// core/orientation.py:40-183).
static std::vector<std::array<int, 3>> feature_order()
{
    std::vector<std::array<int, 3>> faces, edges, corners;
    for (int a = -1; a <= 1; a++)
        for (int b = -1; b <= 1; b++)
            for (int c = -1; c <= 1; c++) {
                const int s = abs(a) + abs(b) + abs(c);
                if (s == 1)
                    faces.push_back({a, b, c});
                else if (s == 2)
                    edges.push_back({a, b, c});
            }
    for (int a : {-1, 1})
        for (int b : {-1, 1})
            for (int c : {-1, 1})
                corners.push_back({a, b, c});
    std::vector<std::array<int, 3>> all = faces;
    all.insert(all.end(), edges.begin(), edges.end());
    all.insert(all.end(), corners.begin(), corners.end());
    return all;
}

// One periodic feature's seam: its own and neighbour slabs and the opposite
// feature's neighbour and own slabs they pair with, row by row.
struct SeamFeature {
    Box own, nb, oown, onb;
    long long rows;
};

// Every feature's distinct seam keys (label << 32 | twin label) in order of
// first row, one feature at a time: keys in row order, stable radix sort,
// first row of every distinct key.  Two host round trips per feature.
template <class Src>
static int seam_keys_each(const Src &src, const std::vector<SeamFeature> &fs,
                          std::vector<std::vector<uint64_t>> &out, cudaStream_t st)
{
    out.assign(fs.size(), {});
    for (size_t fi = 0; fi < fs.size(); fi++) {
        const SeamFeature &f = fs[fi];
        const long long rows = f.rows;
        uint64_t *d_k = nullptr, *d_k2 = nullptr, *d_k3 = nullptr;
        uint32_t *d_i = nullptr, *d_i2 = nullptr;
        uint8_t *d_f = nullptr;
        int *d_nsel = nullptr;
        PMG_TRY(scratch_alloc((void **)&d_k, rows * 8, st));
        PMG_TRY(scratch_alloc((void **)&d_k2, rows * 8, st));
        PMG_TRY(scratch_alloc((void **)&d_k3, rows * 8, st));
        PMG_TRY(scratch_alloc((void **)&d_i, rows * 4, st));
        PMG_TRY(scratch_alloc((void **)&d_i2, rows * 4, st));
        PMG_TRY(scratch_alloc((void **)&d_f, rows, st));
        PMG_TRY(scratch_alloc((void **)&d_nsel, 2 * sizeof(int), st));
        {
            const int ps__ = prof_begin("k_seam_pairs", st);
            k_seam_pairs<Src><<<grid_for(rows, 256, 1LL << 30), 256, 0, st>>>(src, f.own, f.nb, f.onb, f.oown, 0ull,
                                                                            32, 0, d_k, d_i);
            prof_end(ps__, (double)rows * 28, st);
        }
        PMG_CHECK_LAUNCH();
        size_t tb = 0, tb2 = 0, tb3 = 0;
        PMG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, d_k, d_k2, d_i, d_i2, (int)rows, 0, 64, st));
        PMG_CUDA(cub::DeviceSelect::Flagged(nullptr, tb2, d_i2, d_f, d_i, d_nsel, (int)rows, st));
        PMG_CUDA(cub::DeviceSelect::Flagged(nullptr, tb3, d_k2, d_f, d_k3, d_nsel + 1, (int)rows, st));
        size_t tbs = std::max(tb, std::max(tb2, tb3));
        void *d_t = nullptr;
        PMG_TRY(scratch_alloc(&d_t, tbs, st));
        PMG_CUDA(cub::DeviceRadixSort::SortPairs(d_t, tbs, d_k, d_k2, d_i, d_i2, (int)rows, 0, 64, st));
        {
            const int ps__ = prof_begin("k_head_flags", st);
            k_head_flags<<<grid_for(rows, 256, 1LL << 30), 256, 0, st>>>(d_k2, rows, d_f);
            prof_end(ps__, (double)rows * 9, st);
        }
        PMG_CHECK_LAUNCH();
        PMG_CUDA(cub::DeviceSelect::Flagged(d_t, tbs, d_i2, d_f, d_i, d_nsel, (int)rows, st));
        PMG_CUDA(cub::DeviceSelect::Flagged(d_t, tbs, d_k2, d_f, d_k3, d_nsel + 1, (int)rows, st));
        int nsel = 0;
        PMG_CUDA(cudaMemcpyAsync(&nsel, d_nsel, sizeof(int), cudaMemcpyDeviceToHost, st));
        PMG_CUDA(cudaStreamSynchronize(st));
        std::vector<uint32_t> first((size_t)nsel);
        std::vector<uint64_t> dkeys((size_t)nsel);
        if (nsel > 0) {
            PMG_CUDA(cudaMemcpyAsync(first.data(), d_i, (size_t)nsel * 4, cudaMemcpyDeviceToHost, st));
            PMG_CUDA(cudaMemcpyAsync(dkeys.data(), d_k3, (size_t)nsel * 8, cudaMemcpyDeviceToHost, st));
        }
        PMG_CUDA(cudaStreamSynchronize(st));
        for (void *q : {(void *)d_t, (void *)d_k, (void *)d_k2, (void *)d_k3, (void *)d_i, (void *)d_i2, (void *)d_f,
                        (void *)d_nsel})
            PMG_TRY(scratch_free(q, st));
        std::vector<size_t> order((size_t)nsel);
        for (size_t q = 0; q < order.size(); q++)
            order[q] = q;
        std::sort(order.begin(), order.end(), [&](size_t x, size_t y) { return first[x] < first[y]; });
        for (size_t q : order)
            out[fi].push_back(dkeys[q]);
    }
    return PMG_OK;
}

// The same for all features at once, when labels fit `lbits` bits with
// 2 lbits + 5 <= 64: keys (feature << 2 lbits | label << lbits | twin label)
// of every feature in one array, one stable radix sort over those bits, the
// first row of every distinct key; two host round trips in all.  Rows of a
// feature are consecutive and in its row order, so the first row of a key is
// its first occurrence in that feature, as above.
template <class Src>
static int seam_keys_batched(const Src &src, const std::vector<SeamFeature> &fs, int lbits,
                             std::vector<std::vector<uint64_t>> &out, cudaStream_t st)
{
    out.assign(fs.size(), {});
    long long T = 0;
    for (auto &f : fs)
        T += f.rows;
    if (T == 0)
        return PMG_OK;
    if (T >= (1LL << 31)) {
        set_error("periodic merge: %lld seam rows", T);
        return PMG_ERANGE;
    }
    uint64_t *d_k = nullptr, *d_k2 = nullptr, *d_k3 = nullptr;
    uint32_t *d_i = nullptr, *d_i2 = nullptr;
    uint8_t *d_f = nullptr;
    int *d_nsel = nullptr;
    PMG_TRY(scratch_alloc((void **)&d_k, T * 8, st));
    PMG_TRY(scratch_alloc((void **)&d_k2, T * 8, st));
    PMG_TRY(scratch_alloc((void **)&d_k3, T * 8, st));
    PMG_TRY(scratch_alloc((void **)&d_i, T * 4, st));
    PMG_TRY(scratch_alloc((void **)&d_i2, T * 4, st));
    PMG_TRY(scratch_alloc((void **)&d_f, T, st));
    PMG_TRY(scratch_alloc((void **)&d_nsel, 2 * sizeof(int), st));
    {
        const int ps__ = prof_begin("k_seam_pairs", st);
        long long row0 = 0;
        for (size_t fi = 0; fi < fs.size(); fi++) {
            const SeamFeature &f = fs[fi];
            k_seam_pairs<Src><<<grid_for(f.rows, 256, 1LL << 30), 256, 0, st>>>(
                src, f.own, f.nb, f.onb, f.oown, (uint64_t)fi << (2 * lbits), lbits, row0, d_k, d_i);
            row0 += f.rows;
        }
        prof_end(ps__, (double)T * 28, st);
    }
    PMG_CHECK_LAUNCH();
    // rows that repeat the key of the row before cannot be a first row: they go
    // before the sort (labels change rarely along a seam; 12.6 M rows of a
    // 1024^3 field took the sort 0.7 ms)
    const int nbits = 2 * lbits + 5;
    size_t tb = 0, tb2 = 0, tb3 = 0;
    PMG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, d_k, d_k2, d_i, d_i2, (int)T, 0, nbits, st));
    PMG_CUDA(cub::DeviceSelect::Flagged(nullptr, tb2, d_i2, d_f, d_i, d_nsel, (int)T, st));
    PMG_CUDA(cub::DeviceSelect::Flagged(nullptr, tb3, d_k2, d_f, d_k3, d_nsel + 1, (int)T, st));
    size_t tbs = std::max(tb, std::max(tb2, tb3));
    void *d_t = nullptr;
    PMG_TRY(scratch_alloc(&d_t, tbs, st));
    auto heads = [&](const uint64_t *k, long long rows) -> int {
        const int ps__ = prof_begin("k_head_flags", st);
        k_head_flags<<<grid_for(rows, 256, 1LL << 30), 256, 0, st>>>(k, rows, d_f);
        prof_end(ps__, (double)rows * 9, st);
        PMG_CHECK_LAUNCH();
        return PMG_OK;
    };
    int rows = 0;
    PMG_TRY(heads(d_k, T));
    PMG_CUDA(cub::DeviceSelect::Flagged(d_t, tbs, d_i, d_f, d_i2, d_nsel, (int)T, st));
    PMG_CUDA(cub::DeviceSelect::Flagged(d_t, tbs, d_k, d_f, d_k3, d_nsel + 1, (int)T, st));
    PMG_CUDA(cudaMemcpyAsync(&rows, d_nsel, sizeof(int), cudaMemcpyDeviceToHost, st));
    PMG_CUDA(cudaStreamSynchronize(st));
    PMG_CUDA(cub::DeviceRadixSort::SortPairs(d_t, tbs, d_k3, d_k2, d_i2, d_i, rows, 0, nbits, st));
    PMG_TRY(heads(d_k2, rows));
    PMG_CUDA(cub::DeviceSelect::Flagged(d_t, tbs, d_i, d_f, d_i2, d_nsel, rows, st));
    PMG_CUDA(cub::DeviceSelect::Flagged(d_t, tbs, d_k2, d_f, d_k3, d_nsel + 1, rows, st));
    int nsel = 0;
    PMG_CUDA(cudaMemcpyAsync(&nsel, d_nsel, sizeof(int), cudaMemcpyDeviceToHost, st));
    PMG_CUDA(cudaStreamSynchronize(st));
    std::vector<uint32_t> first((size_t)nsel);
    std::vector<uint64_t> dkeys((size_t)nsel);
    if (nsel > 0) {
        PMG_CUDA(cudaMemcpyAsync(first.data(), d_i2, (size_t)nsel * 4, cudaMemcpyDeviceToHost, st));
        PMG_CUDA(cudaMemcpyAsync(dkeys.data(), d_k3, (size_t)nsel * 8, cudaMemcpyDeviceToHost, st));
    }
    PMG_CUDA(cudaStreamSynchronize(st));
    for (void *q : {(void *)d_t, (void *)d_k, (void *)d_k2, (void *)d_k3, (void *)d_i, (void *)d_i2, (void *)d_f,
                    (void *)d_nsel})
        PMG_TRY(scratch_free(q, st));
    // entries come sorted by feature: split, then first-row order per feature
    const uint64_t mask = (1ull << lbits) - 1ull;
    size_t q0 = 0;
    while (q0 < (size_t)nsel) {
        const size_t fi = (size_t)(dkeys[q0] >> (2 * lbits));
        size_t q1 = q0;
        while (q1 < (size_t)nsel && (size_t)(dkeys[q1] >> (2 * lbits)) == fi)
            q1++;
        if (fi >= fs.size()) {
            set_error("periodic merge: bad seam key");
            return PMG_EINVAL;
        }
        std::vector<size_t> order;
        for (size_t q = q0; q < q1; q++)
            order.push_back(q);
        std::sort(order.begin(), order.end(), [&](size_t x, size_t y) { return first[x] < first[y]; });
        for (size_t q : order)
            out[fi].push_back((((dkeys[q] >> lbits) & mask) << 32) | (dkeys[q] & mask));
        q0 = q1;
    }
    return PMG_OK;
}

// Periodic renumbering of the reference (connect_subdomain_boundaries on one
// rank): boundary pairs of every periodic feature, deduplicated on the device
// in first-occurrence order, replayed through the same hash-set container the
// reference uses so its iteration order is reproduced, then the dict / stack
// merge of merge_matched_voxels and local_to_global_labeling on the host
// (boundary data only), and one relabel pass on the device.
// The labels come from src; with lut_out the relabelling table (indexed by
// the local label) is handed back instead of being applied to L.
template <class Src>
static int periodic_renumber(const Src &src, uint64_t *L, const int64_t *shape, const int32_t *bc,
                             const int32_t *pad, int64_t count, int64_t *out_count, cudaStream_t st,
                             uint64_t **lut_out = nullptr)
{
    const long long n = shape[0] * shape[1] * shape[2];
    auto feats = feature_order();
    std::vector<SeamFeature> fs;
    for (auto &f : feats) {
        int fid[3] = {f[0], f[1], f[2]};
        bool has_nb = true;
        int kind = PMG_BC_PERIODIC;
        for (int d = 0; d < 3; d++) {
            if (fid[d] == 0)
                continue;
            const int b = bc[2 * d + (fid[d] > 0 ? 1 : 0)];
            if (b != PMG_BC_PERIODIC)
                has_nb = false;
            if (b == PMG_BC_END)
                kind = PMG_BC_END;
            else if (b == PMG_BC_WALL && kind != PMG_BC_END)
                kind = PMG_BC_WALL;
        }
        if (!has_nb)
            continue;
        int opp[3] = {-fid[0], -fid[1], -fid[2]};
        SeamFeature sf;
        feature_slabs(fid, kind, shape, pad, sf.own, sf.nb);
        feature_slabs(opp, kind, shape, pad, sf.oown, sf.onb);
        sf.rows = sf.own.size() + sf.nb.size();
        if (sf.rows == 0)
            continue;
        if (sf.own.size() != sf.onb.size() || sf.nb.size() != sf.oown.size()) {
            set_error("periodic merge: mismatched feature slabs");
            return PMG_EINVAL;
        }
        fs.push_back(sf);
    }
    // labels (0 .. count) in lbits bits
    int lbits = 1;
    while (lbits < 40 && ((uint64_t)count >> lbits) != 0)
        lbits++;
    std::vector<std::vector<uint64_t>> seam;
    if (2 * lbits + 5 <= 64 && fs.size() <= 32 && tune_value(kTuneCcSeamBatched))
        PMG_TRY(seam_keys_batched(src, fs, lbits, seam, st));
    else
        PMG_TRY(seam_keys_each(src, fs, seam, st));
    // insertion-ordered map (key label -> neighbour list), as a Python dict
    std::vector<uint64_t> keys_order;
    std::vector<std::vector<uint64_t>> nbrs;
    std::unordered_map<uint64_t, long long> key_pos;
    for (auto &keys : seam) {
        // unique_pairs (_voxels.hpp:106-125): the same container fed the same
        // sequence of first insertions iterates in the same order (repeated
        // keys are no-ops)
        std::unordered_set<unsigned long> uset;
        for (uint64_t k : keys)
            uset.insert((unsigned long)k);
        for (unsigned long e : uset) {
            const uint64_t a = e >> 32, b = e & 0xFFFFFFFFul;
            if (a == 0 || b == 0)
                continue;
            // process_matches_by_feature (_voxels.pyx:548-579)
            auto it = key_pos.find(a);
            if (it == key_pos.end()) {
                key_pos.emplace(a, (long long)keys_order.size());
                keys_order.push_back(a);
                nbrs.push_back({b});
            } else {
                auto &lst = nbrs[(size_t)it->second];
                if (std::find(lst.begin(), lst.end(), b) == lst.end())
                    lst.push_back(b);
            }
        }
    }
    // merge_matched_voxels (_voxels.pyx:335-383): stack walk in key order
    std::vector<uint64_t> bl, bg;
    std::vector<char> visited(keys_order.size(), 0);
    uint64_t global_id = 1;
    for (size_t s = 0; s < keys_order.size(); s++) {
        if (visited[s])
            continue;
        std::vector<uint64_t> stack{keys_order[s]};
        std::vector<uint64_t> conns;
        while (!stack.empty()) {
            const uint64_t cur = stack.back();
            stack.pop_back();
            auto it = key_pos.find(cur);
            if (it == key_pos.end()) {
                set_error("periodic merge: neighbour label without a key");
                return PMG_EINVAL;
            }
            if (visited[(size_t)it->second])
                continue;
            visited[(size_t)it->second] = 1;
            conns.push_back(cur);
            for (uint64_t nbl : nbrs[(size_t)it->second]) {
                auto jt = key_pos.find(nbl);
                if (jt == key_pos.end()) {
                    set_error("periodic merge: neighbour label without a key");
                    return PMG_EINVAL;
                }
                if (!visited[(size_t)jt->second])
                    stack.push_back(nbl);
            }
        }
        for (uint64_t c : conns) {
            if (c > (uint64_t)count) {
                set_error("periodic merge: label out of range");
                return PMG_EINVAL;
            }
            bl.push_back(c);
            bg.push_back(global_id);
        }
        global_id += conns.empty() ? 0 : 1;
    }
    // local_to_global_labeling (core/voxels.py:344-397) on the device:
    // boundary labels take their merged id, the others global_id, +1, ...
    // in increasing label order
    const long long m = count + 1;
    const long long nbnd = (long long)bl.size();
    uint64_t *d_lut = nullptr, *d_bl = nullptr, *d_bg = nullptr;
    uint8_t *d_flag = nullptr;
    int *d_nf = nullptr, *d_rank = nullptr;
    PMG_TRY(scratch_alloc((void **)&d_lut, (size_t)m * 8, st));
    PMG_TRY(scratch_alloc((void **)&d_flag, (size_t)m, st));
    PMG_TRY(scratch_alloc((void **)&d_nf, (size_t)m * 4, st));
    PMG_TRY(scratch_alloc((void **)&d_rank, (size_t)m * 4, st));
    PMG_TRY(scratch_alloc((void **)&d_bl, (size_t)(nbnd + 1) * 8, st));
    PMG_TRY(scratch_alloc((void **)&d_bg, (size_t)(nbnd + 1) * 8, st));
    PMG_CUDA(cudaMemsetAsync(d_flag, 0, (size_t)m, st));
    if (nbnd > 0) {
        PMG_CUDA(cudaMemcpyAsync(d_bl, bl.data(), (size_t)nbnd * 8, cudaMemcpyHostToDevice, st));
        PMG_CUDA(cudaMemcpyAsync(d_bg, bg.data(), (size_t)nbnd * 8, cudaMemcpyHostToDevice, st));
        {
            const int ps__ = prof_begin("k_lut_flags", st);
            k_lut_flags<<<grid_for(nbnd, 256, 1LL << 30), 256, 0, st>>>(d_bl, d_bg, nbnd, d_flag, d_lut);
            prof_end(ps__, (double)nbnd * 25, st);
        }
        PMG_CHECK_LAUNCH();
    }
    {
        const int ps__ = prof_begin("k_lut_nonflag", st);
        k_lut_nonflag<<<grid_for(m, 256, 1LL << 30), 256, 0, st>>>(d_flag, m, d_nf);
        prof_end(ps__, (double)m * 5, st);
    }
    PMG_CHECK_LAUNCH();
    size_t tb = 0;
    PMG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, d_nf, d_rank, (int)m, st));
    void *d_t = nullptr;
    PMG_TRY(scratch_alloc(&d_t, tb, st));
    PMG_CUDA(cub::DeviceScan::ExclusiveSum(d_t, tb, d_nf, d_rank, (int)m, st));
    {
        const int ps__ = prof_begin("k_lut_fill", st);
        k_lut_fill<<<grid_for(m, 256, 1LL << 30), 256, 0, st>>>(d_flag, d_rank, m, global_id, d_lut);
        prof_end(ps__, (double)m * 13, st);
    }
    PMG_CHECK_LAUNCH();
    if (!lut_out) {
        const int ps__ = prof_begin("k_apply_lut", st);
        k_apply_lut<<<grid_for(n, 256, 1LL << 30), 256, 0, st>>>(L, n, d_lut);
        prof_end(ps__, (double)n * 16, st);
        PMG_CHECK_LAUNCH();
    }
    const long long nloc = (long long)count - nbnd;
    int64_t max_label = (int64_t)(nloc + (long long)global_id);
    if (max_label < 1)
        max_label = (int64_t)global_id;
    PMG_TRY(scratch_free(d_t, st));
    if (lut_out)
        *lut_out = d_lut;
    else
        PMG_TRY(scratch_free(d_lut, st));
    PMG_TRY(scratch_free(d_flag, st));
    PMG_TRY(scratch_free(d_nf, st));
    PMG_TRY(scratch_free(d_rank, st));
    PMG_TRY(scratch_free(d_bl, st));
    PMG_TRY(scratch_free(d_bg, st));
    *out_count = max_label;
    return PMG_OK;
}

template <typename T>
static int cc_label_t(const T *img, uint64_t *labels, const int64_t *shape, const int32_t *bc,
                      const int32_t *pad, int64_t *count, cudaStream_t st)
{
    const long long n = shape[0] * shape[1] * shape[2];
    int *P = nullptr, *R = nullptr, *err = nullptr, *cnt = nullptr, *offs = nullptr;
    const long long nb = (n + kNumTile - 1) / kNumTile;
    PMG_TRY(scratch_alloc((void **)&P, (size_t)n * 4, st));
    PMG_TRY(scratch_alloc((void **)&R, (size_t)n * 4, st));
    PMG_TRY(scratch_alloc((void **)&err, sizeof(int), st));
    PMG_TRY(scratch_alloc((void **)&cnt, (size_t)nb * 4 + 4, st));
    PMG_TRY(scratch_alloc((void **)&offs, (size_t)nb * 4 + 4, st));
    PMG_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    PMG_TRY(uf_build<T>(img, P, shape, bc, pad, false, err, st));
    {
        const int ps__ = prof_begin("k_root_count", st);
        k_root_count<<<(unsigned)nb, kNumBlock, 0, st>>>(P, n, cnt);
        prof_end(ps__, (double)n * 4, st);
    }
    PMG_CHECK_LAUNCH();
    size_t tb = 0;
    PMG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, offs, (int)nb + 1, st));
    void *tmp = nullptr;
    PMG_TRY(scratch_alloc(&tmp, tb, st));
    PMG_CUDA(cudaMemsetAsync(cnt + nb, 0, 4, st));
    PMG_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, offs, (int)nb + 1, st));
    {
        const int ps__ = prof_begin("k_root_rank", st);
        k_root_rank<<<(unsigned)nb, kNumBlock, 0, st>>>(P, n, offs, R);
        prof_end(ps__, (double)n * 4, st);
    }
    PMG_CHECK_LAUNCH();
    {
        const int ps__ = prof_begin("k_label_out", st);
        k_label_out<<<grid_for(n, 256, 1LL << 30), 256, 0, st>>>(P, R, n, labels);
        prof_end(ps__, (double)n * 12, st);
    }
    PMG_CHECK_LAUNCH();
    int total = 0;
    PMG_CUDA(cudaMemcpyAsync(&total, offs + nb, sizeof(int), cudaMemcpyDeviceToHost, st));
    int s = read_err(err, st);
    PMG_TRY(scratch_free(tmp, st));
    PMG_TRY(scratch_free(P, st));
    PMG_TRY(scratch_free(R, st));
    PMG_TRY(scratch_free(err, st));
    PMG_TRY(scratch_free(cnt, st));
    PMG_TRY(scratch_free(offs, st));
    if (s != PMG_OK)
        return s;
    *count = total;
    if (any_periodic(bc))
        return periodic_renumber(LabImg{labels, Vol3{shape[0], shape[1], shape[2]}}, labels, shape, bc, pad, total,
                                 count, st);
    return PMG_OK;
}

static int check_vol(const int64_t *shape)
{
    for (int d = 0; d < 3; d++)
        if (shape[d] <= 0) {
            set_error("shape[%d] must be positive", d);
            return PMG_EINVAL;
        }
    const long long n = shape[0] * shape[1] * shape[2];
    if (n >= (1LL << 31) - 1) {
        set_error("volume of %lld voxels exceeds the 2^31-1 voxel limit of the int32 union-find", n);
        return PMG_ERANGE;
    }
    return PMG_OK;
}

int cc_label_u8(const uint8_t *img, uint64_t *labels, const int64_t *shape, const int32_t *bc, const int32_t *pad,
                int64_t *count, cudaStream_t st);

} // namespace pmg

using namespace pmg;

extern "C" int pmg_cc_label(const void *img, int32_t elem_bytes, uint64_t *labels,
                            const int64_t shape[3], const int32_t bc[6], const int32_t pad[6],
                            int64_t *count, void *stream)
{
    if (!img || !labels || !shape || !bc || !pad || !count) {
        set_error("pmg_cc_label: null argument");
        return PMG_EINVAL;
    }
    PMG_TRY(check_geometry(shape, bc, pad));
    PMG_TRY(check_vol(shape));
    cudaStream_t st = as_stream(stream);
    switch (elem_bytes) {
    case 1:
        return cc_label_u8((const uint8_t *)img, labels, shape, bc, pad, count, st);
    case 2:
        return cc_label_t((const uint16_t *)img, labels, shape, bc, pad, count, st);
    case 4:
        return cc_label_t((const uint32_t *)img, labels, shape, bc, pad, count, st);
    case 8:
        return cc_label_t((const uint64_t *)img, labels, shape, bc, pad, count, st);
    default:
        set_error("pmg_cc_label: element size %d not supported", elem_bytes);
        return PMG_EINVAL;
    }
}

namespace pmg {

// ---- binary selection on 2x2x2 blocks -----------------------------------------
// When the foreground is a single value (a phase filter, or an image known to
// hold only 0 and 1), all foreground voxels of a 2x2x2 block are mutually
// 26-adjacent and hence in one component, so the union-find runs on blocks:
// eight times fewer elements (the parents of a 512^3 volume fit in L2).  Two
// neighbouring blocks are connected exactly when each has a foreground voxel in
// the part of the block that touches the other (a face, an edge or a corner):
// every voxel of one touching part is 26-adjacent to every voxel of the other.
struct BGrid {
    int s0, s1, s2;    // voxel shape
    int b0, b1, b2;    // block shape
    FastDiv q2, q1;    // division by b2 and by b1
    FastDiv qt;        // division by the pieces of a row (32 blocks)
    // block index -> (c0, c1, c2)
    __device__ __forceinline__ void coords(int b, int &c0, int &c1, int &c2) const
    {
        const int r = (int)fdiv((unsigned)b, q2);
        c2 = b - r * b2;
        c0 = (int)fdiv((unsigned)r, q1);
        c1 = r - c0 * b1;
    }
};

// Foreground of the block selection: the voxels of one value (or nonzero)
// of a uint8 image ...
struct SrcImg {
    const uint8_t *img;
    int fgval;
    // range (optional): OR and AND of the nonzero values seen by the tile pass
    unsigned *range = nullptr;
};

// ... or an erosion read off a capped squared EDT: voxels with E > T stay,
// wall planes are cleared (subtraction + set_wall_bcs,
// morphological_operators.py:171-228).
struct SrcErode {
    const uint16_t *E;
    int T;
    int s0, s1, s2;
    unsigned walls; // bit q: face q (axis q / 2, low / high) is a wall
    __device__ __forceinline__ bool fg(long long idx, int i, int j, int k) const
    {
        const unsigned on = (i == 0) | ((i == s0 - 1) << 1) | ((j == 0) << 2) | ((j == s1 - 1) << 3) |
                            ((k == 0) << 4) | ((k == s2 - 1) << 5);
        return !(on & walls) && (int)E[idx] > T;
    }
    // voxels idx and idx + 1 (idx even, k + 1 < s2) with one 32-bit load
    __device__ __forceinline__ unsigned fg2(long long idx, int i, int j, int k) const
    {
        const unsigned v = *(const uint32_t *)(E + idx);
        const unsigned row = (i == 0) | ((i == s0 - 1) << 1) | ((j == 0) << 2) | ((j == s1 - 1) << 3);
        const unsigned on0 = row | ((k == 0) << 4) | ((k == s2 - 1) << 5);
        const unsigned on1 = row | ((k + 1 == s2 - 1) << 5);
        return (unsigned)(!(on0 & walls) && (int)(v & 0xffffu) > T) |
               ((unsigned)(!(on1 & walls) && (int)(v >> 16) > T) << 1);
    }
};

// ... or the voxels whose step (the first step at which they belong to a
// growing set, 255 for never) is at most k.
struct SrcStep {
    const uint8_t *S;
    int k;
    __device__ __forceinline__ bool fg(long long idx, int, int, int) const { return (int)S[idx] <= k; }
    __device__ __forceinline__ unsigned fg2(long long idx, int, int, int) const
    {
        const unsigned v = *(const uint16_t *)(S + idx);
        return (unsigned)((int)(v & 0xffu) <= k) | ((unsigned)((int)(v >> 8) <= k) << 1);
    }
};

// Mask of block (c0, c1, c2): bit (x * 2 + y) * 2 + z for a foreground voxel
// (2 c0 + x, 2 c1 + y, 2 c2 + z) inside the volume.
template <class Src>
__device__ __forceinline__ unsigned block_mask(const Src &src, const BGrid &G, int c0, int c1, int c2)
{
    unsigned m = 0;
    const long long sy = G.s2, sx = (long long)G.s1 * G.s2;
    const long long base = (2LL * c0 * G.s1 + 2 * c1) * sy + 2 * c2;
    const bool whole = 2 * c0 + 1 < G.s0 && 2 * c1 + 1 < G.s1 && 2 * c2 + 1 < G.s2;
    if (whole && !(G.s2 & 1)) {
        // even rows: every voxel pair (z = 0, 1) starts on an even index
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
            for (int y = 0; y < 2; y++)
                m |= src.fg2(base + x * sx + y * sy, 2 * c0 + x, 2 * c1 + y, 2 * c2) << ((x * 2 + y) * 2);
    } else {
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
            for (int y = 0; y < 2; y++)
#pragma unroll
                for (int z = 0; z < 2; z++) {
                    const int i = 2 * c0 + x, j = 2 * c1 + y, k = 2 * c2 + z;
                    if ((whole || (i < G.s0 && j < G.s1 && k < G.s2)) &&
                        src.fg(base + x * sx + y * sy + z, i, j, k))
                        m |= 1u << ((x * 2 + y) * 2 + z);
                }
    }
    return m;
}

// bytes != 0 -> 0x01 per byte
__device__ __forceinline__ unsigned nonzero01(unsigned v)
{
    return ((((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) >> 7) & 0x01010101u;
}

// The same of an image, its eight bytes in two words; they stay in w for the
// caller (0 outside the volume).
__device__ __forceinline__ unsigned block_mask(const SrcImg &src, const BGrid &G, int c0, int c1, int c2,
                                               unsigned (&w)[2])
{
    const long long sy = G.s2, sx = (long long)G.s1 * G.s2;
    const uint8_t *p = src.img + (2LL * c0 * G.s1 + 2 * c1) * sy + 2 * c2;
    unsigned vol = 0xffu;
    if (2 * c0 + 1 < G.s0 && 2 * c1 + 1 < G.s1 && 2 * c2 + 1 < G.s2 && !(G.s2 & 1)) {
        // even rows: every voxel pair (z = 0, 1) starts on an even index
#pragma unroll
        for (int x = 0; x < 2; x++)
            w[x] = (unsigned)*(const uint16_t *)(p + x * sx) | ((unsigned)*(const uint16_t *)(p + x * sx + sy) << 16);
    } else {
        vol = 0;
        w[0] = w[1] = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int x = q >> 2, y = (q >> 1) & 1, z = q & 1;
            if (2 * c0 + x < G.s0 && 2 * c1 + y < G.s1 && 2 * c2 + z < G.s2) {
                w[x] |= (unsigned)p[x * sx + y * sy + z] << (8 * (q & 3));
                vol |= 1u << q;
            }
        }
    }
    const unsigned pat = src.fgval >= 0 ? (unsigned)src.fgval * 0x01010101u : 0u;
    unsigned a = nonzero01(w[0] ^ pat), b = nonzero01(w[1] ^ pat);
    a = (a | (a >> 7) | (a >> 14) | (a >> 21)) & 0xfu;
    b = (b | (b >> 7) | (b >> 14) | (b >> 21)) & 0xfu;
    const unsigned m = a | (b << 4);
    return (src.fgval >= 0 ? ~m : m) & vol;
}

__device__ __forceinline__ unsigned block_mask(const SrcImg &src, const BGrid &G, int c0, int c1, int c2)
{
    unsigned w[2];
    return block_mask(src, G, c0, c1, c2, w);
}

// OR and AND of the nonzero bytes of a source's voxels, added to its range.
struct ByteRange {
    unsigned o = 0u, a = ~0u;
    __device__ __forceinline__ void add(const unsigned (&w)[2])
    {
        o |= w[0] | w[1];
        a &= (w[0] | (nonzero01(w[0]) ^ 0x01010101u) * 0xffu) & (w[1] | (nonzero01(w[1]) ^ 0x01010101u) * 0xffu);
    }
    // by whole warps
    __device__ __forceinline__ void flush(unsigned *range)
    {
        o |= o >> 16;
        a &= a >> 16;
        o = __reduce_or_sync(0xffffffffu, (o | (o >> 8)) & 0xffu);
        a = __reduce_and_sync(0xffffffffu, (a & (a >> 8)) & 0xffu);
        if ((threadIdx.x & 31) == 0 && o) {
            // (values already seen cost a load)
            if (o & ~*(volatile unsigned *)range)
                atomicOr(range, o);
            if (~a & 0xffu & *(volatile unsigned *)(range + 1))
                atomicAnd(range + 1, a);
        }
    }
};

// Voxels of a block that touch its neighbour at offset (d0, d1, d2): bit
// (x * 2 + y) * 2 + z, x on the d0 side and so on.
__device__ __forceinline__ unsigned touch_bits(int d0, int d1, int d2)
{
    const unsigned X = d0 < 0 ? 0x0Fu : d0 > 0 ? 0xF0u : 0xFFu;
    const unsigned Y = d1 < 0 ? 0x33u : d1 > 0 ? 0xCCu : 0xFFu;
    const unsigned Z = d2 < 0 ? 0x55u : d2 > 0 ? 0xAAu : 0xFFu;
    return X & Y & Z;
}

// ---- row runs -------------------------------------------------------------------
// A tile of 4 x 8 x 32 blocks (8 x 16 x 64 voxels) has 32 rows of 32 blocks along
// the contiguous axis.  A row's masks are kept as eight words, bit c of word i
// the voxel i of block c (one ballot each): touching blocks of a row form
// runs, whose blocks share the first one (the head) as parent, and the
// touching pairs of two neighbouring rows are a few word operations by one
// thread, reduced to one pair per pair of runs before any union.  With a
// block per thread that tested its 13 earlier neighbours and united with a
// cover of them, the two phases were bound by instruction issue (512^3 pack:
// 0.50 and 0.28 ms).

struct RowBits {
    unsigned v[8];
    __device__ __forceinline__ unsigned zlo() const { return v[0] | v[2] | v[4] | v[6]; }
    __device__ __forceinline__ unsigned zhi() const { return v[1] | v[3] | v[5] | v[7]; }
    // blocks that touch the block before them
    __device__ __forceinline__ unsigned runs() const { return zlo() & (zhi() << 1); }
    __device__ __forceinline__ unsigned full() const
    {
        return v[0] & v[1] & v[2] & v[3] & v[4] & v[5] & v[6] & v[7];
    }
    // blocks with one of the voxels `set` among those of even (odd) index
    __device__ __forceinline__ unsigned even(unsigned set) const
    {
        return (set & 1u ? v[0] : 0u) | (set & 4u ? v[2] : 0u) | (set & 16u ? v[4] : 0u) | (set & 64u ? v[6] : 0u);
    }
    __device__ __forceinline__ unsigned odd(unsigned set) const
    {
        return (set & 2u ? v[1] : 0u) | (set & 8u ? v[3] : 0u) | (set & 32u ? v[5] : 0u) | (set & 128u ? v[7] : 0u);
    }
};

__device__ __forceinline__ RowBits row_bits(const unsigned *p) // eight words, 16-byte aligned
{
    const uint4 a = *reinterpret_cast<const uint4 *>(p), b = *reinterpret_cast<const uint4 *>(p + 4);
    return RowBits{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}

// Touching pairs of a row's blocks with the blocks before (em), beside (e0) and
// after (ep) them in neighbouring row q; before, after: the neighbouring
// row's pieces in the tiles beside (their bits 31 and 0 count).
__device__ __forceinline__ void row_pairs(int q, const RowBits &own, const RowBits &nb, const RowBits *before,
                                          const RowBits *after, unsigned &em, unsigned &e0, unsigned &ep)
{
    const int d0 = row_d0(q), d1 = row_d1(q);
    const unsigned a = touch_bits(d0, d1, 0), b = touch_bits(-d0, -d1, 0);
    const unsigned o0 = own.even(a), o1 = own.odd(a), n0 = nb.even(b), n1 = nb.odd(b);
    e0 = (o0 | o1) & (n0 | n1);
    em = o0 & ((n1 << 1) | (before ? before->odd(b) >> 31 : 0u));
    ep = o1 & ((n0 >> 1) | (after ? after->even(b) << 31 : 0u));
}

// words of a block row in the bit array: eight per tile column
__device__ __forceinline__ long long row_word(const BGrid &G, int c0, int c1, int tk, int nt2)
{
    return (((long long)c0 * G.b1 + c1) * nt2 + tk) * 8;
}

// Block masks M and row words V of the source; every later step reads those,
// never the source again.  One warp per piece of a row, lane = block, two pieces
// at a time; bound by the source read.
template <class Src>
__global__ void __launch_bounds__(256) k_block_words(Src src, uint8_t *__restrict__ M, unsigned *__restrict__ V, BGrid G,
                                                     int nt2)
{
    const int lane = threadIdx.x & 31, pieces = G.b0 * G.b1 * nt2;
    constexpr int NP = 2;
    [[maybe_unused]] ByteRange range;
    for (int base = NP * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); base < pieces;
         base += NP * ((gridDim.x * blockDim.x) >> 5)) {
        unsigned m[NP];
        int b[NP];
#pragma unroll
        for (int q = 0; q < NP; q++) {
            const int row = (int)fdiv((unsigned)(base + q), G.qt), c0 = (int)fdiv((unsigned)row, G.q1), c1 = row - c0 * G.b1,
                      c2 = (base + q - row * nt2) * kT2 + lane;
            b[q] = base + q < pieces && c2 < G.b2 ? row * G.b2 + c2 : -1;
            m[q] = 0;
            if constexpr (std::is_same<Src, SrcImg>::value) {
                unsigned w[2] = {0u, 0u};
                if (b[q] >= 0)
                    m[q] = block_mask(src, G, c0, c1, c2, w);
                range.add(w);
            } else if (b[q] >= 0) {
                m[q] = block_mask(src, G, c0, c1, c2);
            }
        }
#pragma unroll
        for (int q = 0; q < NP; q++) {
            if (b[q] >= 0)
                M[b[q]] = (uint8_t)m[q];
            unsigned mine = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const unsigned w = __ballot_sync(0xffffffffu, (m[q] >> i) & 1u);
                mine = lane == i ? w : mine;
            }
            if (lane < 8 && base + q < pieces)
                V[(long long)(base + q) * 8 + lane] = mine;
        }
    }
    if constexpr (std::is_same<Src, SrcImg>::value)
        if (src.range)
            range.flush(src.range);
}

// Phase 1: a shared-memory union-find of the tile's row words whose roots are
// the smallest block index of each tile-local part.  Thread 4 r + q makes the
// pairs of row r with its neighbouring row q, then looks up the parents of its
// eight blocks of row r.
// With R, the tile-local roots are also kept as bits (one word per 32 blocks of
// a row): phase 2 only writes the parents of tile roots, so those bits restore
// the parents of a tile that has not changed (dirty: per tile, cleared here).
// A step is a few dependent loads of shared memory, so what counts is the
// tiles in flight: 128 threads a tile keep a dozen of them on an SM.  With the
// masks read and a thread per block (two tiles in flight) this took 2.85 ms at
// 1024^3 (now 0.84 ms for k_block_words and 0.61 ms here), and restoring
// unchanged tiles from a copy of the parents 0.14 ms a radius of the 512^3
// drainage (now 0.03 ms).
constexpr int kTileThreads = 4 * kT0 * kT1;

__global__ void __launch_bounds__(kTileThreads) k_bcc_tile(const unsigned *__restrict__ V, int *__restrict__ P, BGrid G,
                                                        unsigned *__restrict__ R, int *__restrict__ dirty)
{
    __shared__ __align__(16) int L[kTile];
    __shared__ __align__(16) unsigned s_v[kT0 * kT1 * 8];
    const TileId T;
    const int t = threadIdx.x, r = t >> 2, q = t & 3, a = r / kT1, b = r % kT1;
    const int c0 = T.ti * kT0 + a, c1 = T.tj * kT1 + b;
    const bool in_row = c0 < G.b0 && c1 < G.b1;
    const int row = c0 * G.b1 + c1, piece = row * T.nt2 + T.tk, x0 = row * G.b2 + T.tk * kT2;
    if (dirty && !dirty[T.index()]) {
        if (in_row)
            for (unsigned w = R[piece] & (0xffu << (8 * q)); w; w &= w - 1) {
                const int x = x0 + __ffs(w) - 1;
                P[x] = x;
            }
        return;
    }
    reinterpret_cast<uint2 *>(s_v)[t] =
        in_row ? *reinterpret_cast<const uint2 *>(V + (long long)piece * 8 + 2 * q) : make_uint2(0u, 0u);
#pragma unroll
    for (int i = 0; i < kTile / (4 * kTileThreads); i++) {
        const int e = 4 * (t + i * kTileThreads);
        *reinterpret_cast<int4 *>(L + e) = make_int4(e, e + 1, e + 2, e + 3);
    }
    __syncthreads();
    const RowBits own = row_bits(s_v + r * 8);
    const unsigned ca = own.runs();
    const int d0 = row_d0(q), d1 = row_d1(q);
    if (a + d0 >= 0 && b + d1 >= 0 && b + d1 < kT1) {
        const int rn = r + d0 * kT1 + d1;
        const RowBits nb = row_bits(s_v + rn * 8);
        unsigned em, e0, ep;
        row_pairs(q, own, nb, nullptr, nullptr, em, e0, ep);
        if (q > 0 && a > 0) {
            // where the block above and a further neighbour are both full,
            // they touch each other and that union is theirs
            const RowBits up = row_bits(s_v + (r - kT1) * 8);
            const unsigned centre = (own.even(0x0Fu) | own.odd(0x0Fu)) & up.full(), f = nb.full();
            e0 &= ~(centre & f);
            em &= ~(centre & (f << 1));
            ep &= ~(centre & (f >> 1));
        }
        const unsigned cb = nb.runs();
        row_reduce(ca, cb, em, e0, ep);
        while (em | e0 | ep) {
            const int dz = e0 ? 0 : em ? -1 : 1;
            const unsigned e = e0 ? e0 : em ? em : ep;
            const int c = __ffs(e) - 1;
            const unsigned bit = e & (0u - e);
            e0 &= ~(dz == 0 ? bit : 0u);
            em &= ~(dz < 0 ? bit : 0u);
            ep &= ~(dz > 0 ? bit : 0u);
            sunite(L, r * kT2 + run_head(ca, c), rn * kT2 + run_head(cb, c + dz));
        }
    }
    __syncthreads();
    if (in_row) {
        const unsigned some = own.zlo() | own.zhi();
        int out[8], head = -1, root = -1, roots = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int c = 8 * q + i;
            out[i] = -1;
            if ((some >> c) & 1u) {
                const int h = run_head(ca, c);
                if (h != head) {
                    head = h;
                    const int l = sfind(L, r * kT2 + h);
                    roots |= (l == r * kT2 + c) << i;
                    const int ra = l / (kT1 * kT2), rb = (l / kT2) % kT1, rc = l % kT2;
                    root = ((T.ti * kT0 + ra) * G.b1 + T.tj * kT1 + rb) * G.b2 + T.tk * kT2 + rc;
                }
                out[i] = root;
            }
        }
        const int left = G.b2 - T.tk * kT2 - 8 * q; // blocks of the row from here
        int *dst = P + x0 + 8 * q;
        if (left >= 8 && !(G.b2 & 3)) {
            reinterpret_cast<int4 *>(dst)[0] = make_int4(out[0], out[1], out[2], out[3]);
            reinterpret_cast<int4 *>(dst)[1] = make_int4(out[4], out[5], out[6], out[7]);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (i < left)
                    dst[i] = out[i];
        }
        if (R)
            reinterpret_cast<uint8_t *>(R + piece)[q] = (uint8_t)roots;
    }
    if (dirty && t == 0)
        dirty[T.index()] = 0;
}

// Phase 2: unions across tile borders, one thread block per tile and one thread
// per pair of rows in different tiles or per row end, whose slanted (and, at
// the low end, straight) neighbours lie in the tiles beside.
constexpr int kCrossThreads = 128;
static_assert(kCrossPairs + kT0 * kT1 * 2 <= kCrossThreads, "a thread per pair and per row end");

__global__ void __launch_bounds__(kCrossThreads) k_bcc_cross(int *P, const uint8_t *__restrict__ M,
                                                             const unsigned *__restrict__ V, BGrid G, int *err)
{
    __shared__ CrossSet S;
    const TileId T;
    S.init();
    // pairs of blocks: bit c of em, e0, ep is block x + c with y + c - 1, y + c
    // and y + c + 1
    unsigned em = 0, e0 = 0, ep = 0;
    int x = 0, y = 0;
    const int i = threadIdx.x;
    if (i < kCrossPairs) {
        int a, b, q;
        cross_pair(i, a, b, q);
        const int c0 = T.ti * kT0 + a, c1 = T.tj * kT1 + b, n0 = c0 + row_d0(q), n1 = c1 + row_d1(q);
        if (c0 < G.b0 && c1 < G.b1 && n0 >= 0 && n1 >= 0 && n1 < G.b1) {
            const unsigned *nv = V + row_word(G, n0, n1, T.tk, T.nt2);
            const RowBits own = row_bits(V + row_word(G, c0, c1, T.tk, T.nt2)), nb = row_bits(nv);
            RowBits before = {}, after = {};
            if (T.tk > 0)
                before = row_bits(nv - 8);
            if (T.tk + 1 < T.nt2)
                after = row_bits(nv + 8);
            row_pairs(q, own, nb, &before, &after, em, e0, ep);
            row_reduce(own.runs(), nb.runs(), em, e0, ep);
            x = (c0 * G.b1 + c1) * G.b2 + T.tk * kT2;
            y = (n0 * G.b1 + n1) * G.b2 + T.tk * kT2;
        }
    } else if (i >= kCrossThreads - kT0 * kT1 * 2) {
        const int k = i - (kCrossThreads - kT0 * kT1 * 2), r = k >> 1, a = r / kT1, b = r % kT1;
        const bool low = !(k & 1);
        const int dz = low ? -1 : 1;
        const int c0 = T.ti * kT0 + a, c1 = T.tj * kT1 + b, c2 = T.tk * kT2 + (low ? 0 : kT2 - 1);
        const bool in = c0 < G.b0 && c1 < G.b1 && c2 < G.b2 && c2 + dz >= 0 && c2 + dz < G.b2;
        x = (c0 * G.b1 + c1) * G.b2 + c2;
        const unsigned m = in ? M[x] : 0u;
        if (m) {
            // touching neighbours as bits 0-4 (0-3: row q, 4: the block before)
            unsigned todo = 0;
            if (low && (m & touch_bits(0, 0, -1)) && (M[x - 1] & touch_bits(0, 0, 1)))
                todo = 16u;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int d0 = row_d0(q), d1 = row_d1(q);
                if (a + d0 < 0 || b + d1 < 0 || b + d1 >= kT1 || c1 + d1 >= G.b1)
                    continue; // (a row pair's, or outside)
                if ((m & touch_bits(d0, d1, dz)) &&
                    (M[x + (d0 * G.b1 + d1) * G.b2 + dz] & touch_bits(-d0, -d1, -dz)))
                    todo |= 1u << q;
            }
            while (todo) {
                const int q = __ffs(todo) - 1;
                todo &= todo - 1;
                S.add(P, x, q == 4 ? x - 1 : x + (row_d0(q) * G.b1 + row_d1(q)) * G.b2 + dz, err);
            }
        }
    }
    while (em | e0 | ep) {
        const int dz = e0 ? 0 : em ? -1 : 1;
        const unsigned e = e0 ? e0 : em ? em : ep;
        const int c = __ffs(e) - 1;
        const unsigned bit = e & (0u - e);
        e0 &= ~(dz == 0 ? bit : 0u);
        em &= ~(dz < 0 ? bit : 0u);
        ep &= ~(dz > 0 ? bit : 0u);
        S.add(P, x + c, y + c + dz, err);
    }
    S.finish(P, err);
}

// periodic seams at block level: a foreground halo voxel joins the block of the
// own voxel it copies when that voxel is foreground too
__device__ __forceinline__ bool mfg(const uint8_t *__restrict__ M, const BGrid &G, long long i, long long j,
                                    long long k)
{
    const int b = (int)(((i >> 1) * G.b1 + (j >> 1)) * G.b2 + (k >> 1));
    return (M[b] >> ((((int)i & 1) * 2 + ((int)j & 1)) * 2 + ((int)k & 1))) & 1;
}

__global__ void k_bcc_twins(const uint8_t *__restrict__ M, int *P, BGrid G, Twins W, int *err)
{
    const long long n = W.s0 * W.s1 * W.s2;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        long long c[3];
        c[2] = idx % W.s2;
        const long long r = idx / W.s2;
        c[1] = r % W.s1;
        c[0] = r / W.s1;
        bool halo = false, ok = true;
        long long t[3];
        for (int d = 0; d < 3; d++) {
            t[d] = c[d];
            const long long S = d == 0 ? W.s0 : d == 1 ? W.s1 : W.s2;
            if (c[d] < W.own_lo[d] || c[d] >= W.own_lo[d] + W.own_len[d]) {
                if (!W.periodic[d] || W.own_len[d] <= 0 || c[d] >= S) {
                    ok = false;
                } else {
                    long long q = (c[d] - W.own_lo[d]) % W.own_len[d];
                    if (q < 0)
                        q += W.own_len[d];
                    t[d] = q + W.own_lo[d];
                    halo = true;
                }
            }
        }
        if (!halo || !ok || !mfg(M, G, c[0], c[1], c[2]) || !mfg(M, G, t[0], t[1], t[2]))
            continue;
        const int ba = (int)(((c[0] >> 1) * G.b1 + (c[1] >> 1)) * G.b2 + (c[2] >> 1));
        const int bb = (int)(((t[0] >> 1) * G.b1 + (t[1] >> 1)) * G.b2 + (t[2] >> 1));
        // from their parents: only the parents of tile roots are written
        const int pa = ld(P + ba), pb = ld(P + bb);
        if (pa != pb)
            unite(P, pa, pb, err);
    }
}

// two consecutive coordinates v0, v0 + 1 inside [lo, hi): bits 0, 1
__device__ __forceinline__ unsigned in2(int v0, long long lo, long long hi)
{
    return (unsigned)(v0 >= lo && v0 < hi) | ((unsigned)(v0 + 1 >= lo && v0 + 1 < hi) << 1);
}

// per-axis 2-bit masks spread over the block's bit layout (x * 2 + y) * 2 + z
__device__ __forceinline__ unsigned spread_x(unsigned a) { return (a & 1 ? 0x0Fu : 0u) | (a & 2 ? 0xF0u : 0u); }
__device__ __forceinline__ unsigned spread_y(unsigned a) { return (a & 1 ? 0x33u : 0u) | (a & 2 ? 0xCCu : 0u); }
__device__ __forceinline__ unsigned spread_z(unsigned a) { return (a & 1 ? 0x55u : 0u) | (a & 2 ? 0xAAu : 0u); }

// bytes 0 and 1 of a 16-bit pair equal to v: bits 0, 1
__device__ __forceinline__ unsigned eq2(unsigned pair, unsigned v)
{
    return (unsigned)((pair & 0xffu) == v) | ((unsigned)((pair >> 8) == v) << 1);
}

// Marks of the roots of the blocks with a foreground voxel inside the box:
// one thread per block that meets the box.
__global__ void k_bcc_mark(const uint8_t *__restrict__ M, const int *__restrict__ P, BGrid G, Box bx,
                           uint8_t *mark, uint8_t bit, int *err)
{
    long long lo[3], nbk[3];
    for (int d = 0; d < 3; d++) {
        lo[d] = bx.lo[d] >> 1;
        nbk[d] = ((bx.hi[d] + 1) >> 1) - lo[d];
    }
    const long long n = nbk[0] * nbk[1] * nbk[2];
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const int c2 = (int)(lo[2] + q % nbk[2]), c1 = (int)(lo[1] + (q / nbk[2]) % nbk[1]),
                  c0 = (int)(lo[0] + q / (nbk[2] * nbk[1]));
        const int b = (c0 * G.b1 + c1) * G.b2 + c2;
        const unsigned inbox = spread_x(in2(2 * c0, bx.lo[0], bx.hi[0])) & spread_y(in2(2 * c1, bx.lo[1], bx.hi[1])) &
                               spread_z(in2(2 * c2, bx.lo[2], bx.hi[2]));
        if (!(M[b] & inbox))
            continue;
        int p = ld(P + b);
        if (p >= 0)
            p = find_root(P, p, err);
        if (p >= 0 && !(mark[p] & bit))
            atomicOr((unsigned int *)(mark + (p & ~3)), (unsigned int)bit << (8 * (p & 3)));
    }
}

// One thread per block: the block's root and marks decide all its voxels at
// once; kept foreground voxels receive `val`, everything else 0.  A warp
// covers 32 consecutive blocks, i.e. 64 contiguous voxels of each of the
// block's four rows.
template <typename TO>
__global__ void k_bcc_select(const uint8_t *__restrict__ M, int *P, const uint8_t *__restrict__ mark, BGrid G,
                             int mode, TO val, TO *__restrict__ out, unsigned long long *kept, int *err)
{
    const int nb = G.b0 * G.b1 * G.b2;
    unsigned int cnt = 0; // kept voxels (mask bits exist only for voxels inside the volume)
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        int c0, c1, c2;
        G.coords(b, c0, c1, c2);
        unsigned m = M[b];
        if (m) {
            // the root, and the parent flattened to it
            int p = ld(P + b);
            if (p >= 0 && p != b) {
                const int q = find_root(P, p, err);
                if (q != p)
                    P[b] = q;
                p = q;
            }
            const uint8_t mk = p >= 0 ? mark[p] : 0;
            const bool in = mk & 1, ou = mk & 2;
            bool keep;
            if (mode == PMG_SEL_INLET)
                keep = in;
            else if (mode == PMG_SEL_OUTLET)
                keep = ou;
            else if (mode == PMG_SEL_BOTH)
                keep = in && ou;
            else
                keep = !(in || ou);
            if (!keep)
                m = 0;
        }
        cnt += __popc(m);
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
            for (int y = 0; y < 2; y++) {
                const int i = 2 * c0 + x, j = 2 * c1 + y;
                if (i >= G.s0 || j >= G.s1)
                    continue;
                TO *row = out + ((long long)i * G.s1 + j) * G.s2;
#pragma unroll
                for (int z = 0; z < 2; z++) {
                    const int k = 2 * c2 + z;
                    if (k < G.s2)
                        row[k] = ((m >> ((x * 2 + y) * 2 + z)) & 1) ? val : (TO)0;
                }
            }
    }
    if (kept) {
        for (int o = 16; o > 0; o >>= 1)
            cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        if ((threadIdx.x & 31) == 0 && cnt)
            atomicAdd(kept, (unsigned long long)cnt);
    }
}

__host__ __device__ inline const uint8_t *src_elem(const SrcImg &s) { return s.img; }
__host__ __device__ inline const uint16_t *src_elem(const SrcErode &s) { return s.E; }
__host__ __device__ inline const uint8_t *src_elem(const SrcStep &s) { return s.S; }
// bytes a tile pass reads from its source: one element per voxel, or one mask per block
template <class Src>
static double src_bytes(const Src &src, long long n, long long nb)
{
    return (double)n * sizeof(*src_elem(src));
}

static BGrid bgrid_of(const int64_t *shape)
{
    BGrid G;
    G.s0 = (int)shape[0];
    G.s1 = (int)shape[1];
    G.s2 = (int)shape[2];
    G.b0 = (G.s0 + 1) / 2;
    G.b1 = (G.s1 + 1) / 2;
    G.b2 = (G.s2 + 1) / 2;
    G.q2 = fastdiv_of((unsigned)G.b2);
    G.q1 = fastdiv_of((unsigned)G.b1);
    G.qt = fastdiv_of((unsigned)((G.b2 + kT2 - 1) / kT2));
    return G;
}

// bytes of the row words of a block grid
static size_t bcc_row_bytes(const BGrid &G)
{
    return (size_t)G.b0 * G.b1 * (size_t)((G.b2 + kT2 - 1) / kT2) * 8 * sizeof(unsigned);
}

static dim3 bcc_tiles(const BGrid &G)
{
    return dim3((unsigned)((G.b2 + kT2 - 1) / kT2), (unsigned)((G.b1 + kT1 - 1) / kT1),
                (unsigned)((G.b0 + kT0 - 1) / kT0));
}

// Phase 1 from the row words; dirty: of the flagged tiles alone, the others'
// parents being restored (R of an earlier call).
static int bcc_tiles_run(const int64_t *shape, int *P, const unsigned *V, unsigned *R, int *dirty, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const int ps__ = prof_begin("k_bcc_tile", st);
    k_bcc_tile<<<bcc_tiles(G), kTileThreads, 0, st>>>(V, P, G, R, dirty);
    prof_end(ps__, (double)G.b0 * G.b1 * G.b2 * (dirty ? 1.0 / 8 : 5.0), st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// Masks, row words (V: bcc_row_bytes) and phase 1 of the block union-find.
template <class Src>
static int bcc_tile_phase(const Src &src, const int64_t *shape, int *P, uint8_t *M, unsigned *V, cudaStream_t st,
                          unsigned *R = nullptr)
{
    const BGrid G = bgrid_of(shape);
    const int nb = G.b0 * G.b1 * G.b2, nt2 = (G.b2 + kT2 - 1) / kT2;
    const long long pieces = (long long)G.b0 * G.b1 * nt2;
    const int ps__ = prof_begin("k_block_words", st);
    k_block_words<Src><<<grid_for((pieces + 1) / 2 * 32, 256, 152LL * 64), 256, 0, st>>>(src, M, V, G, nt2);
    prof_end(ps__, src_bytes(src, (long long)shape[0] * shape[1] * shape[2], nb) + (double)nb * 2, st);
    PMG_CHECK_LAUNCH();
    return bcc_tiles_run(shape, P, V, R, nullptr, st);
}

// Phase 2 and the periodic seams (twins).
static int bcc_cross_phase(const int64_t *shape, const int32_t *bc, const int32_t *pad, bool twins, int *P,
                           const uint8_t *M, const unsigned *V, int *err, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const long long n = shape[0] * shape[1] * shape[2];
    const dim3 tiles = bcc_tiles(G);
    {
        const int ps__ = prof_begin("k_bcc_cross", st);
        k_bcc_cross<<<tiles, kCrossThreads, 0, st>>>(P, M, V, G, err);
        // the words of the rows of every pair
        prof_end(ps__, (double)tiles.x * tiles.y * tiles.z * kCrossPairs * 2 * kT2, st);
        PMG_CHECK_LAUNCH();
    }
    if (twins && any_periodic(bc)) {
        const int ps__ = prof_begin("k_bcc_twins", st);
        k_bcc_twins<<<grid_for(n, 256, 152LL * 32), 256, 0, st>>>(M, P, G, make_twins(shape, bc, pad), err);
        prof_end(ps__, 0.0, st);
        PMG_CHECK_LAUNCH();
    }
    return PMG_OK;
}

// Block union-find of the source: tiles, cross-tile unions, periodic seams
// (twins).  P[b]: a parent on the way to the root block (the smallest block
// index of the component), -1 for empty blocks; M[b] = block mask.
template <class Src>
static int bcc_build(const Src &src, const int64_t *shape, const int32_t *bc, const int32_t *pad, bool twins,
                     int *P, uint8_t *M, int *err, cudaStream_t st, unsigned *Vkeep = nullptr,
                     unsigned *R = nullptr)
{
    unsigned *V = Vkeep;
    if (!V)
        PMG_TRY(scratch_alloc((void **)&V, bcc_row_bytes(bgrid_of(shape)), st));
    int s = bcc_tile_phase(src, shape, P, M, V, st, R);
    if (s == PMG_OK)
        s = bcc_cross_phase(shape, bc, pad, twins, P, M, V, err, st);
    if (!Vkeep)
        PMG_TRY(scratch_free(V, st));
    return s;
}

// Inlet / outlet boxes (lo0, hi0, lo1, hi1, lo2, hi2; null or lo0 < 0 for
// none) must lie inside the volume.
static int check_boxes(const int64_t *shape, const int64_t *inlet_box, const int64_t *outlet_box)
{
    const int64_t *boxes[2] = {inlet_box, outlet_box};
    for (int w = 0; w < 2; w++) {
        const int64_t *bxp = boxes[w];
        if (!bxp || bxp[0] < 0)
            continue;
        for (int d = 0; d < 3; d++)
            if (bxp[2 * d] < 0 || bxp[2 * d + 1] > shape[d] || bxp[2 * d] > bxp[2 * d + 1]) {
                set_error("connected-image selection: face box outside the volume");
                return PMG_EINVAL;
            }
    }
    return PMG_OK;
}

// Marks of the roots of blocks with foreground in the inlet (bit 0) and
// outlet (bit 1) boxes; parents need not be flat.
static int bcc_marks(const int64_t *shape, const int64_t *inlet_box, const int64_t *outlet_box, const int *P,
                     const uint8_t *M, uint8_t *mark, int *err, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const int nb = G.b0 * G.b1 * G.b2;
    PMG_CUDA(cudaMemsetAsync(mark, 0, ((size_t)nb + 3) & ~(size_t)3, st));
    const int64_t *boxes[2] = {inlet_box, outlet_box};
    for (int w = 0; w < 2; w++) {
        const int64_t *bxp = boxes[w];
        if (!bxp || bxp[0] < 0)
            continue;
        Box b;
        for (int d = 0; d < 3; d++) {
            b.lo[d] = bxp[2 * d];
            b.hi[d] = bxp[2 * d + 1];
        }
        if (b.size() > 0) {
            long long nbk = 1;
            for (int d = 0; d < 3; d++)
                nbk *= ((b.hi[d] + 1) >> 1) - (b.lo[d] >> 1);
            const int ps__ = prof_begin("k_bcc_mark", st);
            k_bcc_mark<<<grid_for(nbk, 256, 1LL << 30), 256, 0, st>>>(M, P, G, b, mark, (uint8_t)(1 << w), err);
            // per block meeting the box: mask, parent, root parent
            prof_end(ps__, (double)nbk * 9, st);
            PMG_CHECK_LAUNCH();
        }
    }
    return PMG_OK;
}

// The selection from parents P (flattened on the way), masks M and marks.
static int bcc_select_out(void *out, int out_bytes, const int64_t *shape, int mode, int val, int *P,
                          const uint8_t *M, const uint8_t *mark, int *err, cudaStream_t st,
                          unsigned long long *kept)
{
    const BGrid G = bgrid_of(shape);
    const int nb = G.b0 * G.b1 * G.b2;
    const long long n = shape[0] * shape[1] * shape[2];
    const int ps__ = prof_begin("k_bcc_select", st);
    if (out_bytes == 1)
        k_bcc_select<uint8_t><<<grid_for(nb, 256, 152LL * 64), 256, 0, st>>>(M, P, mark, G, mode, (uint8_t)val,
                                                                           (uint8_t *)out, kept, err);
    else
        k_bcc_select<uint64_t><<<grid_for(nb, 256, 152LL * 64), 256, 0, st>>>(M, P, mark, G, mode, (uint64_t)val,
                                                                            (uint64_t *)out, kept, err);
    prof_end(ps__, (double)n * out_bytes + (double)nb * 5, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

static int bcc_mark_select(void *out, int out_bytes, const int64_t *shape, const int64_t *inlet_box,
                           const int64_t *outlet_box, int mode, int val, int *P, const uint8_t *M, uint8_t *mark,
                           int *err, cudaStream_t st, unsigned long long *kept)
{
    PMG_TRY(bcc_marks(shape, inlet_box, outlet_box, P, M, mark, err, st));
    return bcc_select_out(out, out_bytes, shape, mode, val, P, M, mark, err, st, kept);
}

template <class Src>
static int bcc_select_core(const Src &src, void *out, int out_bytes, const int64_t *shape, const int32_t *bc,
                           const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box, int mode,
                           int val, int *P, uint8_t *M, uint8_t *mark, int *err, cudaStream_t st,
                           unsigned long long *kept)
{
    PMG_TRY(check_boxes(shape, inlet_box, outlet_box));
    PMG_TRY(bcc_build(src, shape, bc, pad, true, P, M, err, st));
    return bcc_mark_select(out, out_bytes, shape, inlet_box, outlet_box, mode, val, P, M, mark, err, st, kept);
}

// Binary selection: P and mark need one int / one byte per 2x2x2 block.  Kept
// voxels receive `fgval`, or 1 for fgval < 0 (an image of 0s and 1s).
int select_run_binary(const uint8_t *img, void *out, int out_bytes, const int64_t *shape, const int32_t *bc,
                      const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box, int mode,
                      int fgval, int *P, uint8_t *M, uint8_t *mark, int *err, cudaStream_t st,
                      unsigned long long *kept)
{
    SrcImg src{img, fgval};
    return bcc_select_core(src, out, out_bytes, shape, bc, pad, inlet_box, outlet_box, mode, fgval >= 0 ? fgval : 1,
                           P, M, mark, err, st, kept);
}

// Erosion fused into the selection: the foreground is E > T off the wall
// planes, with E a capped squared EDT (uint16, units of res^2) of the
// unextended image; kept voxels receive 1.
int select_run_erode(const uint16_t *E, int T, void *out, const int64_t *shape, const int32_t *bc,
                     const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box, int mode, int *P,
                     uint8_t *M, uint8_t *mark, int *err, cudaStream_t st, unsigned long long *kept)
{
    SrcErode src;
    src.E = E;
    src.T = T;
    src.s0 = (int)shape[0];
    src.s1 = (int)shape[1];
    src.s2 = (int)shape[2];
    src.walls = 0;
    for (int q = 0; q < 6; q++)
        src.walls |= (bc[q] == PMG_BC_WALL ? 1u : 0u) << q;
    return bcc_select_core(src, out, 1, shape, bc, pad, inlet_box, outlet_box, mode, 1, P, M, mark, err, st, kept);
}

// ---- selection of a growing set -----------------------------------------------
// Along a drainage curve two selected sets only ever grow: the eroded pore
// space (its threshold falls with the radius) and the non-wetting phase (the
// update turns wetting voxels non-wetting, never back).  Components of a
// growing set only merge, so after one full block union-find a step unites the
// touching pairs with a block that changed (N, one bit per block); every other
// pair is in one component already.  And a block once connected to the inlet
// stays so: where the step's selection (k_pair_rows) takes the connected blocks
// out of U (one bit per block), later steps neither look up their roots nor
// unite two of them.  What a step keeps true of any two touching blocks is
// "same component, or both connected": an equivalence, so pairs that the row
// reduction leaves out follow from those that it keeps.

struct GrowWords {
    unsigned *V, *N, *U;
};

// A block's new mask m: masks, row words, the changed and unconnected bits and,
// for a block that was empty, its own root.  A mask that lost voxels is an
// error (code 3): the set did not grow.
__device__ __forceinline__ void grow_block(const BGrid &G, int b, int c0, int c1, int c2, unsigned old, unsigned m,
                                           uint8_t *M, int *P, const GrowWords &W, int nt2, int *err)
{
    if (m == old)
        return;
    if (old & ~m)
        atomicExch(err, 3);
    M[b] = (uint8_t)m;
    const long long piece = row_word(G, c0, c1, c2 / kT2, nt2) / 8;
    const unsigned bit = 1u << (c2 % kT2);
    if (!old) {
        P[b] = b;
        atomicOr(W.U + piece, bit);
    }
    atomicOr(W.N + piece, bit);
    for (unsigned delta = m & ~old; delta; delta &= delta - 1)
        atomicOr(W.V + piece * 8 + __ffs(delta) - 1, bit);
}

template <class Src>
__global__ void k_grow_masks(Src src, uint8_t *M, int *P, GrowWords W, BGrid G, int nt2,
                             int *err)
{
    const int nb = G.b0 * G.b1 * G.b2;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        // the old mask and the source are loaded independently
        int c2, c0, c1;
        G.coords(b, c0, c1, c2);
        const unsigned old = M[b];
        grow_block(G, b, c0, c1, c2, old, block_mask(src, G, c0, c1, c2), M, P, W, nt2, err);
    }
}

// Listed blocks (steps known in advance) take their masks from the source.
template <class Src>
__global__ void k_grow_apply(Src src, uint8_t *M, int *P, GrowWords W, BGrid G, int nt2,
                             const int *__restrict__ list, const int *__restrict__ off, int *err,
                             unsigned long long *units)
{
    const int a = off[0], cnt = off[1] - a;
    if (units && blockIdx.x == 0 && threadIdx.x == 0 && cnt > 0)
        atomicAdd(units, (unsigned long long)cnt);
    for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < cnt; it += gridDim.x * blockDim.x) {
        const int b = list[a + it];
        int c2, c0, c1;
        G.coords(b, c0, c1, c2);
        const unsigned old = M[b];
        grow_block(G, b, c0, c1, c2, old, block_mask(src, G, c0, c1, c2), M, P, W, nt2, err);
    }
}

// After the full union-find: every block unconnected, none changed.
__global__ void k_grow_start(GrowWords W, int pieces)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < pieces; q += gridDim.x * blockDim.x) {
        const RowBits r = row_bits(W.V + (long long)q * 8);
        W.U[q] = r.zlo() | r.zhi();
        W.N[q] = 0u;
    }
}

// The unions of a step: the
// touching pairs of a row piece (32 blocks) within the row and with the four
// earlier neighbouring rows that have a changed block and an unconnected one.
// A thread per piece and neighbouring row (and one for the pairs within the
// row) lists them: the changed and unconnected words, 1/8 of the row words, tell
// most of the threads that there are none.  k_grow_join then unites them, a
// thread per pair: a union is a chain of dependent loads, so it is taken off
// the threads that are mostly idle.
// Bound by those chains.  A warp per grown block with a lane per neighbour spent
// 0.28 ms a radius of the 512^3 drainage on three dependent loads per block and
// on unions of blocks that were in one component already, a thread per piece and
// row that united its own pairs 0.15 ms with half as many pairs (0.60 ms where
// most pairs were new); now 0.09 ms for the list and 0.10 ms for the unions.
struct RowSet {
    int *P;
    GrowWords W;
    int2 *list;
    int *count;
    int cap; // pairs beyond it are united at once
};
constexpr int kGrowPieces = 32, kGrowThreads = 5 * kGrowPieces;

__global__ void __launch_bounds__(kGrowThreads) k_grow_pairs(RowSet R, BGrid G, int nt2, int *err)
{
    const GrowWords W = R.W;
    const int q = threadIdx.x / kGrowPieces, piece = blockIdx.x * kGrowPieces + threadIdx.x % kGrowPieces;
    const int row = (int)fdiv((unsigned)piece, G.qt), tk = piece - row * nt2;
    const int c0 = (int)fdiv((unsigned)row, G.q1), c1 = row - c0 * G.b1;
    // q < 4: neighbouring row q; q == 4: the row itself (its blocks before)
    const int d0 = q < 4 ? row_d0(q) : 0, d1 = q < 4 ? row_d1(q) : 0;
    bool work = piece < G.b0 * G.b1 * nt2 && c0 + d0 >= 0 && c1 + d1 >= 0 && c1 + d1 < G.b1;
    const int o = piece + (d0 * G.b1 + d1) * nt2;
    unsigned n = 0, u = 0, nn = 0, un = 0, nm = 0, um = 0, n1 = 0, u1 = 0;
    if (work) {
        n = W.N[piece];
        u = W.U[piece];
        nn = W.N[o];
        un = W.U[o];
        if (tk > 0) {
            nm = W.N[o - 1];
            um = W.U[o - 1];
        }
        if (q < 4 && tk + 1 < nt2) {
            n1 = W.N[o + 1];
            u1 = W.U[o + 1];
        }
        work = (n | nn | nm | n1) && (u | un | um | u1);
    }
    if (!__any_sync(0xffffffffu, work))
        return;
    // bits of the pairs with the blocks before, beside and after
    unsigned em = 0, e0 = 0, ep = 0;
    if (work) {
        const RowBits own = row_bits(W.V + (long long)piece * 8);
        const unsigned cz = own.runs();
        if (q == 4) {
            em = cz;
            if (tk > 0)
                em |= own.zlo() & (row_bits(W.V + (long long)(piece - 1) * 8).zhi() >> 31);
        } else {
            const unsigned *nv = W.V + (long long)o * 8;
            const RowBits nb = row_bits(nv);
            RowBits before = {}, after = {};
            if (tk > 0)
                before = row_bits(nv - 8);
            if (tk + 1 < nt2)
                after = row_bits(nv + 8);
            row_pairs(q, own, nb, &before, &after, em, e0, ep);
            row_reduce(cz, nb.runs(), em, e0, ep);
        }
        em &= (n | nn << 1 | nm >> 31) & (u | un << 1 | um >> 31);
        e0 &= (n | nn) & (u | un);
        ep &= (n | nn >> 1 | n1 << 31) & (u | un >> 1 | u1 << 31);
    }
    // the warp's pairs take consecutive entries
    const int lane = threadIdx.x & 31, mine = __popc(em) + __popc(e0) + __popc(ep);
    int at = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, d);
        at += lane >= d ? v : 0;
    }
    int first = 0;
    if (lane == 31 && at)
        first = atomicAdd(R.count, at);
    at += __shfl_sync(0xffffffffu, first, 31) - mine;
    const int x = row * G.b2 + tk * kT2, y = x + (d0 * G.b1 + d1) * G.b2;
    while (em | e0 | ep) {
        const int dz = e0 ? 0 : em ? -1 : 1;
        const unsigned f = e0 ? e0 : em ? em : ep;
        const int c = __ffs(f) - 1;
        const unsigned bit = f & (0u - f);
        e0 &= ~(dz == 0 ? bit : 0u);
        em &= ~(dz < 0 ? bit : 0u);
        ep &= ~(dz > 0 ? bit : 0u);
        if (at < R.cap)
            R.list[at] = make_int2(x + c, y + c + dz);
        else
            unite(R.P, x + c, y + c + dz, err);
        at++;
    }
}

// The listed pairs united; the roots that a block of threads joins are mostly
// the same few (CrossSet).
__global__ void __launch_bounds__(256) k_grow_join(RowSet R, int *err, unsigned long long *units)
{
    __shared__ CrossSet S;
    const int n = min(*R.count, R.cap);
    if (units && blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(units, (unsigned long long)n);
    if ((int)(blockIdx.x * blockDim.x) >= n)
        return;
    S.init();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int2 e = R.list[k];
        S.join(R.P, e.x, e.y, err);
    }
}

static int row_pieces(const BGrid &G) { return G.b0 * G.b1 * ((G.b2 + kT2 - 1) / kT2); }

static size_t piece_bytes(const BGrid &G) { return ((size_t)row_pieces(G) * 4 + 255) & ~(size_t)255; }

size_t grow_sel_bytes(const int64_t *shape)
{
    const BGrid G = bgrid_of(shape);
    const size_t nb = (size_t)G.b0 * G.b1 * G.b2;
    const size_t a = (nb + 255) & ~(size_t)255;
    // parents, masks, marks, row words, changed and unconnected words, pairs
    return a * 4 + a + a + bcc_row_bytes(G) + 2 * piece_bytes(G) + a * 4 + 256;
}

void grow_sel_init(GrowSel &g, void *mem, const int64_t *shape)
{
    const BGrid G = bgrid_of(shape);
    const size_t nb = (size_t)G.b0 * G.b1 * G.b2;
    const size_t a = (nb + 255) & ~(size_t)255;
    char *p = (char *)mem;
    g.P = (int *)p;
    p += a * 4;
    g.M = (uint8_t *)p;
    p += a;
    g.mark = (uint8_t *)p;
    p += a;
    g.V = (unsigned *)p;
    p += bcc_row_bytes(G);
    g.N = (unsigned *)p;
    p += piece_bytes(G);
    g.U = (unsigned *)p;
    p += piece_bytes(G);
    g.pairs = (int2 *)p;
    g.npairs = (int *)(p + a * 4);
    g.built = false;
}

static GrowWords words(const GrowSel &g) { return GrowWords{g.V, g.N, g.U}; }

// The set's first step: the full block union-find.
template <class Src>
static int grow_build(GrowSel &g, const Src &src, const int64_t *shape, const int32_t *bc, const int32_t *pad, int *err,
                      cudaStream_t st)
{
    PMG_TRY(bcc_build(src, shape, bc, pad, true, g.P, g.M, err, st, g.V));
    const int pieces = row_pieces(bgrid_of(shape));
    const int ps__ = prof_begin("k_grow_start", st);
    k_grow_start<<<grid_for(pieces, 256, 152LL * 16), 256, 0, st>>>(words(g), pieces);
    prof_end(ps__, (double)pieces * 40, st);
    PMG_CHECK_LAUNCH();
    PMG_CUDA(cudaMemsetAsync(g.npairs, 0, sizeof(int), st));
    g.stamp = 0;
    g.built = true;
    g.pending = false;
    return PMG_OK;
}

// The set's masks and row words brought up to date: from its list of step off,
// or from the source, or (pending) by the producer already.
template <class Src>
static int grow_masks(GrowSel &g, const Src &src, const int64_t *shape, const int *off, int *err, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const int nb = G.b0 * G.b1 * G.b2, nt2 = (G.b2 + kT2 - 1) / kT2;
    if (off) {
        const int ps__ = prof_begin("k_grow_apply", st);
        k_grow_apply<Src><<<152 * 8, 256, 0, st>>>(src, g.M, g.P, words(g), G, nt2, g.ev, off, err,
                                                   prof_units(kUnitsGrowApply));
        // per listed block: its list entry, eight source elements, mask read
        // and written, parent written
        prof_end_units(ps__, kUnitsGrowApply, 4 + 8 * sizeof(*src_elem(src)) + 2 + 4, st);
    } else if (!g.pending) {
        const int ps__ = prof_begin("k_grow_masks", st);
        k_grow_masks<Src><<<grid_for(nb, 256, 152LL * 64), 256, 0, st>>>(src, g.M, g.P, words(g), G, nt2, err);
        prof_end(ps__, (double)shape[0] * shape[1] * shape[2] * sizeof(*src_elem(src)) + (double)nb, st);
    }
    PMG_CHECK_LAUNCH();
    g.pending = false;
    return PMG_OK;
}

// The step's unions (the pair count is zero: the selection of the last step or
// the build cleared it).
static int grow_rows(GrowSel &g, const int64_t *shape, int *err, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const int nt2 = (G.b2 + kT2 - 1) / kT2, pieces = row_pieces(G), cap = G.b0 * G.b1 * G.b2 / 2;
    const RowSet R{g.P, words(g), g.pairs, g.npairs, cap};
    {
        const int ps__ = prof_begin("k_grow_pairs", st);
        k_grow_pairs<<<(unsigned)((pieces + kGrowPieces - 1) / kGrowPieces), kGrowThreads, 0, st>>>(R, G, nt2, err);
        // the changed and the unconnected words (the words of pieces with pairs come on top)
        prof_end(ps__, (double)pieces * 8, st);
    }
    PMG_CHECK_LAUNCH();
    {
        const int ps__ = prof_begin("k_grow_join", st);
        k_grow_join<<<(unsigned)grid_for(cap, 256, 152LL * 4), 256, 0, st>>>(R, err, prof_units(kUnitsGrowJoin));
        // per pair: its entry, both blocks' parents and a root's
        prof_end_units(ps__, kUnitsGrowJoin, 8 + 3 * 4, st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// One step of a growing selection up to the marks.
template <class Src>
static int grow_step(GrowSel &g, const Src &src, const int64_t *shape, const int32_t *bc, const int32_t *pad,
                     const int64_t *inlet_box, const int64_t *outlet_box, int *err, cudaStream_t st)
{
    PMG_TRY(check_boxes(shape, inlet_box, outlet_box));
    if (!g.built) {
        PMG_TRY(grow_build(g, src, shape, bc, pad, err, st));
    } else {
        PMG_TRY(grow_masks(g, src, shape, nullptr, err, st));
        PMG_TRY(grow_rows(g, shape, err, st));
        PMG_CUDA(cudaMemsetAsync(g.N, 0, piece_bytes(bgrid_of(shape)), st));
        PMG_CUDA(cudaMemsetAsync(g.npairs, 0, sizeof(int), st));
        if (any_periodic(bc)) {
            const BGrid G = bgrid_of(shape);
            const long long n = shape[0] * shape[1] * shape[2];
            const int ps__ = prof_begin("k_bcc_twins", st);
            k_bcc_twins<<<grid_for(n, 256, 152LL * 32), 256, 0, st>>>(g.M, g.P, G, make_twins(shape, bc, pad), err);
            prof_end(ps__, 0.0, st);
            PMG_CHECK_LAUNCH();
        }
    }
    g.stamp = 0; // the marks below are no stamps
    return bcc_marks(shape, inlet_box, outlet_box, g.P, g.M, g.mark, err, st);
}

template <class Src>
static int grow_select_core(GrowSel &g, const Src &src, void *out, const int64_t *shape, const int32_t *bc,
                            const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box, int mode,
                            int val, int *err, cudaStream_t st, unsigned long long *kept)
{
    PMG_TRY(grow_step(g, src, shape, bc, pad, inlet_box, outlet_box, err, st));
    return bcc_select_out(out, 1, shape, mode, val, g.P, g.M, g.mark, err, st, kept);
}

static SrcErode erode_src(const uint16_t *E, int T, const int64_t *shape, const int32_t *bc)
{
    SrcErode src;
    src.E = E;
    src.T = T;
    src.s0 = (int)shape[0];
    src.s1 = (int)shape[1];
    src.s2 = (int)shape[2];
    src.walls = 0;
    for (int q = 0; q < 6; q++)
        src.walls |= (bc[q] == PMG_BC_WALL ? 1u : 0u) << q;
    return src;
}

// Marks by stamp: the roots of the set's blocks with a voxel in the box get this
// step's stamp, so that the marks of earlier steps
// need no clearing.
struct StampSet {
    const uint8_t *M;
    int *P;
    uint8_t *mark;
    uint8_t stamp;
};

__global__ void k_face_stamp(StampSet R, BGrid G, Box bx, int *err)
{
    int lo[3], nbk[3];
    for (int d = 0; d < 3; d++) {
        lo[d] = (int)(bx.lo[d] >> 1);
        nbk[d] = (int)((bx.hi[d] + 1) >> 1) - lo[d];
    }
    const int n = nbk[0] * nbk[1] * nbk[2];
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int c2 = lo[2] + q % nbk[2], c1 = lo[1] + (q / nbk[2]) % nbk[1], c0 = lo[0] + q / (nbk[2] * nbk[1]);
        const int b = (c0 * G.b1 + c1) * G.b2 + c2;
        const unsigned inbox = spread_x(in2(2 * c0, bx.lo[0], bx.hi[0])) & spread_y(in2(2 * c1, bx.lo[1], bx.hi[1])) &
                               spread_z(in2(2 * c2, bx.lo[2], bx.hi[2]));
        if (!(R.M[b] & inbox))
            continue;
        int p = ld(R.P + b);
        if (p >= 0 && p != b)
            p = find_root(R.P, p, err);
        if (p >= 0 && R.mark[p] != R.stamp)
            R.mark[p] = R.stamp;
    }
}

// The next stamp of a mark array (cleared when the stamps run out).
static int next_stamp(uint8_t *mark, int &stamp, size_t nb, cudaStream_t st)
{
    if (stamp == 0 || stamp == 255) {
        PMG_CUDA(cudaMemsetAsync(mark, 0, nb, st));
        stamp = 0;
    }
    stamp++;
    return PMG_OK;
}

static int face_stamps(const int64_t *box, const int64_t *shape, StampSet R, int *err, cudaStream_t st)
{
    if (!box || box[0] < 0)
        return PMG_OK;
    Box b;
    long long nbk = 1;
    for (int d = 0; d < 3; d++) {
        b.lo[d] = box[2 * d];
        b.hi[d] = box[2 * d + 1];
        nbk *= ((b.hi[d] + 1) >> 1) - (b.lo[d] >> 1);
    }
    if (b.size() <= 0)
        return PMG_OK;
    const int ps__ = prof_begin("k_face_stamp", st);
    k_face_stamp<<<(unsigned)grid_for(nbk, 128, 1LL << 30), 128, 0, st>>>(R, bgrid_of(shape), b, err);
    // per block meeting the box: mask, parent, root parent
    prof_end(ps__, (double)nbk * 9, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// Inlet selection of set A constrained by set B, as row words: the voxels of A
// whose component has the inlet stamp and, when *b_count > 0, that are voxels
// of B with the inlet stamp too (porosimetry.py:130-148: img_results kept
// where n_connected == 1 once the phase exists); kept counts A's
// inlet-connected voxels before the constraint, xr receives the block-plane
// range of the output (kRangeBig encoding).  A warp takes four pieces of a row,
// lane 8 q + i holding word i of piece q.  Only unconnected blocks' roots are
// looked up (lane = block, the four pieces' loads of each level before any of
// them is used, because they are chains of dependent loads), their parents
// being flattened on the way; what is connected now leaves U, and the changed
// bits are cleared.
// Bound by the three row words read and written per piece where most blocks
// are connected (0.08 ms a radius of the 512^3 drainage; with a root lookup for
// every block 0.14 ms).
struct SelectSet {
    const uint8_t *mark;
    int *P;
    uint8_t stamp;
    GrowWords W;
    int *npairs; // cleared for the next step
};

// The unconnected blocks of four pieces (u: each lane its piece's) looked up;
// what stays unconnected.
__device__ __forceinline__ unsigned still_unconnected(const SelectSet &A, unsigned u, int piece0, int nt2,
                                                      const BGrid &G, int *err)
{
    constexpr int NB = 4;
    const int lane = threadIdx.x & 31;
    int x[NB], p[NB], g[NB];
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const int row = (int)fdiv((unsigned)(piece0 + q), G.qt);
        x[q] = row * G.b2 + (piece0 + q - row * nt2) * kT2 + lane;
        p[q] = (__shfl_sync(0xffffffffu, u, q * 8) >> lane) & 1u ? ld(A.P + x[q]) : -1;
    }
#pragma unroll
    for (int q = 0; q < NB; q++)
        g[q] = p[q] >= 0 && p[q] != x[q] ? ld(A.P + p[q]) : p[q];
#pragma unroll
    for (int q = 0; q < NB; q++)
        if (g[q] != p[q]) {
            p[q] = find_root(A.P, g[q], err);
            A.P[x[q]] = p[q];
        }
    bool k[NB];
#pragma unroll
    for (int q = 0; q < NB; q++)
        k[q] = p[q] >= 0 && A.mark[p[q]] == A.stamp;
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const unsigned got = __ballot_sync(0xffffffffu, k[q]);
        if ((lane >> 3) == q)
            u &= ~got;
    }
    return u;
}

__global__ void __launch_bounds__(256) k_pair_rows(SelectSet A, SelectSet B,
                                                   const unsigned long long *__restrict__ b_count, BGrid G, int nt2,
                                                   unsigned *__restrict__ out, unsigned long long *kept, int *err,
                                                   int *xr)
{
    const int pieces = G.b0 * G.b1 * nt2, lane = threadIdx.x & 31;
    const bool constrain = *b_count > 0;
    unsigned cnt = 0;
    int xmax = 0, xmin = 0;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *A.npairs = *B.npairs = 0;
    for (int base = warp * 4; base < pieces; base += nwarps * 4) {
        const int piece = base + (lane >> 3);
        const bool in = piece < pieces;
        const long long word = (long long)base * 8 + lane;
        const unsigned va = in ? A.W.V[word] : 0u, vb = in && constrain ? B.W.V[word] : 0u;
        const unsigned ua0 = in ? A.W.U[piece] : 0u, ub0 = in ? B.W.U[piece] : 0u;
        unsigned ua = ua0, ub = ub0;
        if (__any_sync(0xffffffffu, ua0))
            ua = still_unconnected(A, ua0, base, nt2, G, err);
        if (__any_sync(0xffffffffu, ub0))
            ub = still_unconnected(B, ub0, base, nt2, G, err);
        if (in && (lane & 7) == 0) {
            if (ua != ua0)
                A.W.U[piece] = ua;
            if (ub != ub0)
                B.W.U[piece] = ub;
            A.W.N[piece] = 0u;
            B.W.N[piece] = 0u;
        }
        const unsigned wa = va & ~ua, o = constrain ? wa & vb & ~ub : wa;
        cnt += __popc(wa);
        if (in)
            out[word] = o;
        if (o) {
            const int c0 = (int)fdiv(fdiv((unsigned)piece, G.qt), G.q1);
            xmax = max(xmax, c0 + 1);
            xmin = max(xmin, kRangeBig - c0);
        }
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    xmax = __reduce_max_sync(0xffffffffu, xmax);
    xmin = __reduce_max_sync(0xffffffffu, xmin);
    if (lane == 0) {
        if (cnt)
            atomicAdd(kept, (unsigned long long)cnt);
        if (xmax) {
            atomicMax(xr, xmax);
            atomicMax(xr + 1, xmin);
        }
    }
}

// Step values (255 outside the volume) of the eight voxels of a block, byte
// (x * 2 + y) * 2 + z of the result.
__device__ __forceinline__ unsigned long long block_steps(const uint8_t *S, const BGrid &G, int c0, int c1, int c2)
{
    unsigned long long v = ~0ull;
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
        for (int y = 0; y < 2; y++) {
            const int i = 2 * c0 + x, j = 2 * c1 + y, k = 2 * c2;
            if (i >= G.s0 || j >= G.s1)
                continue;
            const long long a = ((long long)i * G.s1 + j) * G.s2 + k;
            unsigned pair;
            if (!(G.s2 & 1))
                pair = *(const uint16_t *)(S + a);
            else
                pair = S[a] | (k + 1 < G.s2 ? (unsigned)S[a + 1] << 8 : 0xff00u);
            const int sh = 8 * ((x * 2 + y) * 2);
            v = (v & ~(0xffffull << sh)) | ((unsigned long long)pair << sh);
        }
    return v;
}

// Distinct steps < nsteps among a block's eight voxels, packed in the low
// bytes of the result; their number in nd.
__device__ __forceinline__ unsigned long long distinct_steps(unsigned long long v, int nsteps, int &nd)
{
    unsigned long long d = 0;
    nd = 0;
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int x = (int)((v >> (8 * e)) & 0xffu);
        bool fresh = x < nsteps;
#pragma unroll
        for (int f = 0; f < e; f++)
            fresh = fresh && x != (int)((v >> (8 * f)) & 0xffu);
        if (fresh) {
            d |= (unsigned long long)x << (8 * nd);
            nd++;
        }
    }
    return d;
}

// Per-step counters live 32 ints apart (separate cache lines, separate L2
// slices).
constexpr int kStepStride = 32;

// Events (block, step) for every distinct step of a block: counted per step
// in shared memory, then added to the global counters once per CTA.
__global__ void k_step_count(const uint8_t *__restrict__ S, BGrid G, int nsteps, int *cnt)
{
    __shared__ int hist[256];
    for (int v = threadIdx.x; v < 256; v += blockDim.x)
        hist[v] = 0;
    __syncthreads();
    const int nb = G.b0 * G.b1 * G.b2;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        int c0, c1, c2, nd;
        G.coords(b, c0, c1, c2);
        const unsigned long long d = distinct_steps(block_steps(S, G, c0, c1, c2), nsteps, nd);
        for (int e = 0; e < nd; e++)
            atomicAdd(&hist[(d >> (8 * e)) & 0xffu], 1);
    }
    __syncthreads();
    for (int v = threadIdx.x; v < nsteps; v += blockDim.x)
        if (hist[v])
            atomicAdd(cnt + v * kStepStride, hist[v]);
}

// The events written at per-step cursors: each round of blockDim.x blocks
// counts its events per step in shared memory, reserves one range per step
// with a single global atomic, then writes them.
__global__ void k_step_scatter(const uint8_t *__restrict__ S, BGrid G, int nsteps, int *cursor, int *__restrict__ ev)
{
    __shared__ int hist[256];
    __shared__ int sbase[256];
    for (int v = threadIdx.x; v < 256; v += blockDim.x)
        hist[v] = 0;
    __syncthreads();
    const int nb = G.b0 * G.b1 * G.b2;
    for (int base = blockIdx.x * blockDim.x; base < nb; base += gridDim.x * blockDim.x) {
        const int b = base + threadIdx.x;
        int nd = 0;
        unsigned long long d = 0;
        int loc[8];
        if (b < nb) {
            int c0, c1, c2;
            G.coords(b, c0, c1, c2);
            d = distinct_steps(block_steps(S, G, c0, c1, c2), nsteps, nd);
        }
#pragma unroll
        for (int e = 0; e < 8; e++)
            loc[e] = e < nd ? atomicAdd(&hist[(d >> (8 * e)) & 0xffu], 1) : 0;
        __syncthreads();
        for (int v = threadIdx.x; v < nsteps; v += blockDim.x) {
            sbase[v] = hist[v] ? atomicAdd(cursor + v * kStepStride, hist[v]) : 0;
            hist[v] = 0;
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (e < nd)
                ev[sbase[(d >> (8 * e)) & 0xffu] + loc[e]] = b;
    }
}

// Exclusive prefix of the per-step counts into the offsets (off[nsteps] =
// total), the cursors reset to the offsets; one thread block.
__global__ void k_step_offsets(int *cnt_cursor, int nsteps, int *off)
{
    if (threadIdx.x == 0) {
        int total = 0;
        for (int k = 0; k < nsteps; k++) {
            const int c = cnt_cursor[k * kStepStride];
            off[k] = total;
            cnt_cursor[k * kStepStride] = total;
            total += c;
        }
        off[nsteps] = total;
    }
}

int step_lists_build(GrowSel &g, const uint8_t *S, const int64_t *shape, int nsteps, void **mem, cudaStream_t st)
{
    *mem = nullptr;
    if (nsteps <= 0 || nsteps > 255) {
        set_error("step lists: %d steps outside [1, 255]", nsteps);
        return PMG_EINVAL;
    }
    const BGrid G = bgrid_of(shape);
    const int nb = G.b0 * G.b1 * G.b2;
    // a block has at most min(8, nsteps) distinct steps: the list is sized for
    // that, so nothing has to be read back before the scatter
    const size_t cap = (size_t)nb * (size_t)(nsteps < 8 ? nsteps : 8);
    const size_t tmpb = sizeof(int) * (size_t)kStepStride * 256;
    const size_t offb = ((size_t)(nsteps + 1) * sizeof(int) + 255) & ~(size_t)255;
    char *m = nullptr;
    PMG_TRY(scratch_alloc((void **)&m, tmpb + offb + sizeof(int) * cap, st));
    int *tmp = (int *)m;
    g.off = (int *)(m + tmpb);
    g.ev = (int *)(m + tmpb + offb);
    *mem = m;
    PMG_CUDA(cudaMemsetAsync(tmp, 0, tmpb, st));
    {
        const int ps__ = prof_begin("k_step_count", st);
        k_step_count<<<grid_for(nb, 256, 152LL * 8), 256, 0, st>>>(S, G, nsteps, tmp);
        prof_end(ps__, (double)nb * 8, st);
    }
    PMG_CHECK_LAUNCH();
    k_step_offsets<<<1, 32, 0, st>>>(tmp, nsteps, g.off);
    PMG_CHECK_LAUNCH();
    {
        const int ps__ = prof_begin("k_step_scatter", st);
        k_step_scatter<<<grid_for(nb, 256, 152LL * 8), 256, 0, st>>>(S, G, nsteps, tmp, g.ev);
        prof_end(ps__, (double)nb * 8, st);
    }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

template <class Src>
static int grow_marks(GrowSel &g, const Src &src, const int64_t *shape, const int32_t *bc, const int32_t *pad,
                      const int *off, const int64_t *inlet_box, int *err, cudaStream_t st)
{
    PMG_TRY(check_boxes(shape, inlet_box, nullptr));
    if (!g.built) {
        PMG_TRY(grow_build(g, src, shape, bc, pad, err, st));
    } else {
        PMG_TRY(grow_masks(g, src, shape, off, err, st));
        PMG_TRY(grow_rows(g, shape, err, st));
    }
    const BGrid G = bgrid_of(shape);
    PMG_TRY(next_stamp(g.mark, g.stamp, (size_t)G.b0 * G.b1 * G.b2, st));
    return face_stamps(inlet_box, shape, StampSet{g.M, g.P, g.mark, (uint8_t)g.stamp}, err, st);
}

int grow_marks_eroded(GrowSel &g, const uint8_t *S, int k, const uint16_t *E, int T, const int64_t *shape,
                      const int32_t *bc, const int32_t *pad, const int64_t *inlet_box, int *err, cudaStream_t st)
{
    return S ? grow_marks(g, SrcStep{S, k}, shape, bc, pad, g.ev ? g.off + k : nullptr, inlet_box, err, st)
             : grow_marks(g, erode_src(E, T, shape, bc), shape, bc, pad, nullptr, inlet_box, err, st);
}

int grow_marks_phase(GrowSel &g, const uint8_t *img, int fgval, const int64_t *shape, const int32_t *bc,
                     const int32_t *pad, const int64_t *inlet_box, int *err, cudaStream_t st)
{
    return grow_marks(g, SrcImg{img, fgval}, shape, bc, pad, nullptr, inlet_box, err, st);
}

int grow_pair_select(GrowSel &a, GrowSel &b, const unsigned long long *b_count, unsigned *out, const int64_t *shape,
                     int *err, cudaStream_t st, unsigned long long *kept, int *xr)
{
    const BGrid G = bgrid_of(shape);
    const int pieces = row_pieces(G);
    const int ps__ = prof_begin("k_pair_rows", st);
    k_pair_rows<<<grid_for((pieces + 3) / 4 * 32LL, 256, 152LL * 32), 256, 0, st>>>(
        SelectSet{a.mark, a.P, (uint8_t)a.stamp, words(a), a.npairs},
        SelectSet{b.mark, b.P, (uint8_t)b.stamp, words(b), b.npairs}, b_count, G,
        (G.b2 + kT2 - 1) / kT2, out, kept, err, xr);
    // words read and written, the unconnected and the changed words (the
    // lookups come on top)
    prof_end(ps__, (double)pieces * (96 + 8 + 8), st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

size_t rows_bytes(const int64_t *shape) { return bcc_row_bytes(bgrid_of(shape)); }

// Row words of the voxels equal to 1 of an image: one warp per piece of a row.
__global__ void __launch_bounds__(256) k_bytes_to_rows(const uint8_t *__restrict__ img, unsigned *__restrict__ V,
                                                       BGrid G, int nt2)
{
    const int lane = threadIdx.x & 31, pieces = G.b0 * G.b1 * nt2;
    const SrcImg src{img, 1};
    for (int piece = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; piece < pieces;
         piece += (gridDim.x * blockDim.x) >> 5) {
        const int row = (int)fdiv((unsigned)piece, G.qt), c0 = (int)fdiv((unsigned)row, G.q1), c1 = row - c0 * G.b1,
                  c2 = (piece - row * nt2) * kT2 + lane;
        const unsigned m = c2 < G.b2 ? block_mask(src, G, c0, c1, c2) : 0u;
        unsigned mine = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const unsigned w = __ballot_sync(0xffffffffu, (m >> i) & 1u);
            mine = lane == i ? w : mine;
        }
        if (lane < 8)
            V[(long long)piece * 8 + lane] = mine;
    }
}

int bytes_to_rows(const uint8_t *img, unsigned *V, const int64_t *shape, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const int pieces = row_pieces(G);
    const int ps__ = prof_begin("k_bytes_to_rows", st);
    k_bytes_to_rows<<<grid_for(pieces * 32LL, 256, 152LL * 32), 256, 0, st>>>(img, V, G, (G.b2 + kT2 - 1) / kT2);
    prof_end(ps__, (double)shape[0] * shape[1] * shape[2] + (double)pieces * 32, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

int select_grow_binary(GrowSel &g, const uint8_t *img, int fgval, void *out, const int64_t *shape,
                       const int32_t *bc, const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box,
                       int mode, int *err, cudaStream_t st, unsigned long long *kept)
{
    SrcImg src{img, fgval};
    return grow_select_core(g, src, out, shape, bc, pad, inlet_box, outlet_box, mode, fgval >= 0 ? fgval : 1, err,
                            st, kept);
}

// ---- selection of a shrinking set, tile by tile ---------------------------------
// The wetting phase of a drainage curve only loses voxels; components can
// split, so its union-find is rebuilt every step, but the tile phase is local:
// a tile none of whose voxels changed gives the same tile-local parents as
// before.  The producer of the changes (the drainage update) flags the tiles it
// touched and keeps the block masks and row words current.

size_t shrink_sel_bytes(const int64_t *shape)
{
    const BGrid G = bgrid_of(shape);
    const size_t nb = (size_t)G.b0 * G.b1 * G.b2;
    const size_t a = (nb + 255) & ~(size_t)255;
    const size_t nt = (size_t)((G.b0 + kT0 - 1) / kT0) * ((G.b1 + kT1 - 1) / kT1) * ((G.b2 + kT2 - 1) / kT2);
    // P, M, mark, per-tile flags, row words, tile roots, cut-off blocks
    return a * 4 + a * 2 + ((nt * 4 + 255) & ~(size_t)255) + bcc_row_bytes(G) + 2 * piece_bytes(G) + 256;
}

void shrink_sel_init(ShrinkSel &g, void *mem, const int64_t *shape)
{
    const BGrid G = bgrid_of(shape);
    const size_t nb = (size_t)G.b0 * G.b1 * G.b2;
    const size_t a = (nb + 255) & ~(size_t)255;
    const size_t nt = (size_t)((G.b0 + kT0 - 1) / kT0) * ((G.b1 + kT1 - 1) / kT1) * ((G.b2 + kT2 - 1) / kT2);
    char *p = (char *)mem;
    g.P = (int *)p;
    p += a * 4;
    g.M = (uint8_t *)p;
    p += a;
    g.mark = (uint8_t *)p;
    p += a;
    g.dirty = (int *)p;
    p += (nt * 4 + 255) & ~(size_t)255;
    g.V = (unsigned *)p;
    p += bcc_row_bytes(G);
    g.R = (unsigned *)p;
    p += piece_bytes(G);
    g.T = (unsigned *)p;
    g.ntiles = (int)nt;
    g.stamp = 0;
    g.built = false;
}

int shrink_marks_binary(ShrinkSel &g, const uint8_t *img, int fgval, const int64_t *shape, const int32_t *bc,
                        const int32_t *pad, const int64_t *outlet_box, int *err, cudaStream_t st)
{
    PMG_TRY(check_boxes(shape, nullptr, outlet_box));
    const BGrid G = bgrid_of(shape);
    if (g.built) {
        PMG_TRY(bcc_tiles_run(shape, g.P, g.V, g.R, g.dirty, st));
        PMG_TRY(bcc_cross_phase(shape, bc, pad, true, g.P, g.M, g.V, err, st));
    } else {
        PMG_CUDA(cudaMemsetAsync(g.dirty, 0, sizeof(int) * (size_t)g.ntiles, st));
        PMG_CUDA(cudaMemsetAsync(g.T, 0, piece_bytes(G), st));
        const SrcImg src{img, fgval};
        PMG_TRY(bcc_build(src, shape, bc, pad, true, g.P, g.M, err, st, g.V, g.R));
    }
    g.built = true;
    PMG_TRY(next_stamp(g.mark, g.stamp, (size_t)G.b0 * G.b1 * G.b2, st));
    return face_stamps(outlet_box, shape, StampSet{g.M, g.P, g.mark, (uint8_t)g.stamp}, err, st);
}

// ---- drainage update on row words -------------------------------------------------
// mp = 1 where morph == 1 on a wetting voxel (2) connected to the outlet,
// reservoir slabs -> 1 (equilibrium_distribution.py:133-179,
// subdomain_padded.py:285-307), fused with the saturation counts (value 2
// inside the own box, multiphase.py:56-96; value 1 anywhere).  Dilation, wetting
// and non-wetting phase are row words, so the image itself is only written,
// where it changes.  A thread per word finds the pieces of a row (32 blocks)
// whose dilation meets wetting voxels not known to be cut off, which are then
// taken by a warp each (lanes 0-7 its words, then lane = block).  The outlet
// connection comes from the wetting phase's block union-find.  The masks and
// words of both phases are kept current, and the wetting phase's changed tiles
// flagged.
// Bound by the words read where little changes, by the root searches elsewhere:
// 0.08 ms a radius at 512^3; a thread per block that read image and dilation byte
// by byte took 0.25 ms, four pieces to a warp one after the other 0.16 ms.

// bit c: position 2 (32 tk + c) + z inside [lo, hi)
__device__ __forceinline__ unsigned range_bits(int tk, int z, long long lo, long long hi)
{
    // positions v = base + 2 c
    const long long base = 64LL * tk + z;
    const long long a = lo > base ? (lo - base + 1) >> 1 : 0, b = hi > base ? (hi - base + 1) >> 1 : 0;
    const unsigned ma = a >= 32 ? 0u : 0xffffffffu << a, mb = b >= 32 ? 0xffffffffu : (1u << b) - 1u;
    return ma & mb;
}

constexpr int kUpdatePieces = 64; // per block of 256 threads

// The running totals (own voxels of value 2, voxels of value 1) from the counts
// of one update, which are cleared, and the saturation numerator.
__device__ __forceinline__ void drain_totals(const DrainCounts &C, int full)
{
    // (atomics: the counts are the other blocks' atomic adds)
    const unsigned long long c2 = atomicExch(C.cnt2, 0ull), c1 = atomicExch(C.cnt1, 0ull);
    *C.tot = full ? c2 : *C.tot - c2;
    *C.ones += c1;
    *C.sat = *C.tot;
}

__global__ void k_drain_same(DrainCounts C) // a radius that changes nothing
{
    *C.sat = *C.tot;
}


struct UpdateSets {
    // wetting phase: row words, masks, parents, outlet stamps, tile flags
    unsigned *Vw;
    uint8_t *Mw;
    int *Pw;
    const uint8_t *markw;
    uint8_t stamp;
    int *wdirty;
    // its blocks found cut off from the outlet (they stay so), one bit each
    unsigned *Tw;
    // non-wetting phase (Vn null: not kept)
    unsigned *Vn, *Nn, *Un;
    uint8_t *Mn;
    int *Pn;
};

// D: the dilation (defined on the block planes of orange; null: none).  full:
// every piece, with the reservoir slabs, the counts being all voxels of value
// 2 in the own box and the voxels newly 1; otherwise only the dilation's planes
// (the slabs were refilled before), and the changes of both counts.
__global__ void __launch_bounds__(256) k_drain_update_rows(uint8_t *__restrict__ mp, const unsigned *__restrict__ D,
                                                           UpdateSets U, BGrid G, int nt2, Boxes B,
                                                           DrainCounts C, int *err, const int *__restrict__ orange,
                                                           int full, unsigned long long *units)
{
    const int bxlo = orange ? orange[0] >> 1 : 0, bxhi = orange ? orange[1] >> 1 : G.b0 - 1;
    const int plane = G.b1 * nt2;
    const int first = full ? 0 : max(0, bxlo) * plane,
              last = full ? G.b0 * plane : min(G.b0 * plane, max(0, bxhi + 1) * plane);
    if (units && blockIdx.x == 0 && threadIdx.x == 0 && last > first)
        atomicAdd(units, (unsigned long long)(last - first) * 256ull);
    const int lane = threadIdx.x & 31, i = lane & 7;
    const int X = i >> 2, Y = (i >> 1) & 1, Z = i & 1; // the voxel of this lane's word
    const long long sx = (long long)G.s1 * G.s2, sy = G.s2;
    unsigned c2n = 0, c1n = 0;
    __shared__ int s_list[kUpdatePieces];
    __shared__ int s_n;
    for (int chunk = first + blockIdx.x * kUpdatePieces; chunk < last; chunk += gridDim.x * kUpdatePieces) {
        if (threadIdx.x == 0)
            s_n = 0;
        __syncthreads();
        for (int p = threadIdx.x >> 3; p < kUpdatePieces; p += blockDim.x >> 3) {
            const int piece = chunk + p;
            unsigned s = 0;
            if (piece < last) {
                const int c0 = (int)fdiv(fdiv((unsigned)piece, G.qt), G.q1);
                if (D && c0 >= bxlo && c0 <= bxhi)
                    s = U.Vw[(long long)piece * 8 + i] & D[(long long)piece * 8 + i] & ~U.Tw[piece];
            }
            const unsigned some = __ballot_sync(0xffffffffu, s != 0);
            if (i == 0 && piece < last && (full || ((some >> (lane & 24)) & 0xffu)))
                s_list[atomicAdd(&s_n, 1)] = piece;
        }
        __syncthreads();
        for (int it = threadIdx.x >> 5; it < s_n; it += blockDim.x >> 5) {
            const int piece = s_list[it];
            const int row = (int)fdiv((unsigned)piece, G.qt), tk = piece - row * nt2;
            const int c0 = (int)fdiv((unsigned)row, G.q1), c1 = row - c0 * G.b1;
            const long long word = (long long)piece * 8 + i;
            const bool in = lane < 8;
            const unsigned w = in ? U.Vw[word] : 0u;
            unsigned set1 = 0;
            if (D && c0 >= bxlo && c0 <= bxhi) {
                set1 = in ? w & D[word] & ~U.Tw[piece] : 0u;
                const unsigned cand = __reduce_or_sync(0xffffffffu, set1);
                int r = -1;
                if ((cand >> lane) & 1u)
                    r = find_root(U.Pw, row * G.b2 + tk * kT2 + lane, err);
                const unsigned on = __ballot_sync(0xffffffffu, r >= 0 && U.markw[r] == U.stamp);
                set1 &= on;
                if (lane == 0 && (cand & ~on))
                    U.Tw[piece] |= cand & ~on;
            }
            if (!full && !__any_sync(0xffffffffu, set1))
                continue;
            const int vi = 2 * c0 + X, vj = 2 * c1 + Y;
            const bool row_in = vi < G.s0 && vj < G.s1;
            const bool own_row = vi >= B.own[0] && vi < B.own[1] && vj >= B.own[2] && vj < B.own[3];
            const unsigned own = in && own_row ? range_bits(tk, Z, B.own[4], B.own[5]) : 0u;
            unsigned fresh = set1; // voxels that were not 1
            if (full) {
                // the reservoir slabs
                const unsigned vol = in && row_in ? range_bits(tk, Z, 0, G.s2) : 0u;
                const bool slab = vi < B.rpad[0] || vi >= G.s0 - B.rpad[1] || vj < B.rpad[2] || vj >= G.s1 - B.rpad[3];
                const unsigned res = slab ? vol : vol & ~range_bits(tk, Z, B.rpad[4], (long long)G.s2 - B.rpad[5]);
                unsigned was1 = 0;
                for (unsigned q = res & ~set1; q; q &= q - 1) {
                    const int c = __ffs(q) - 1;
                    if (mp[vi * sx + vj * sy + 2 * (tk * kT2 + c) + Z] == 1)
                        was1 |= 1u << c;
                }
                set1 |= res;
                fresh = set1 & ~was1;
                c2n += __popc(w & ~set1 & own);
            } else {
                c2n += __popc(set1 & own);
            }
            c1n += __popc(fresh);
            const unsigned any = __reduce_or_sync(0xffffffffu, set1);
            if (!any)
                continue;
            const unsigned nw = in && U.Vn ? U.Vn[word] : 0u;
            const unsigned w2 = w & ~set1, nw2 = nw | set1;
            if (in && set1) {
                U.Vw[word] = w2;
                if (U.Vn)
                    U.Vn[word] = nw2;
            }
            // lane = block: the changed blocks' masks, and the image
            unsigned mw = 0, mn = 0, ms = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                mw |= ((__shfl_sync(0xffffffffu, w2, q) >> lane) & 1u) << q;
                mn |= ((__shfl_sync(0xffffffffu, nw2, q) >> lane) & 1u) << q;
                ms |= ((__shfl_sync(0xffffffffu, set1, q) >> lane) & 1u) << q;
            }
            // blocks of the non-wetting phase that grew and that are new
            const unsigned grown = __reduce_or_sync(0xffffffffu, nw2 & ~nw),
                           fresh_blocks = __reduce_or_sync(0xffffffffu, nw2) & ~__reduce_or_sync(0xffffffffu, nw);
            const bool lost = __any_sync(0xffffffffu, w2 != w);
            if (ms) {
                const int c2 = tk * kT2 + lane, b = row * G.b2 + c2;
                U.Mw[b] = (uint8_t)mw;
                if (U.Vn) {
                    U.Mn[b] = (uint8_t)mn;
                    if ((fresh_blocks >> lane) & 1u)
                        U.Pn[b] = b;
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const unsigned bits = (ms >> (2 * q)) & 3u;
                    uint8_t *p = mp + (2 * c0 + (q >> 1)) * sx + (2 * c1 + (q & 1)) * sy + 2 * c2;
                    if (bits == 3u && !(G.s2 & 1)) {
                        *reinterpret_cast<uint16_t *>(p) = 0x0101u;
                    } else {
                        if (bits & 1u)
                            p[0] = 1;
                        if (bits & 2u)
                            p[1] = 1;
                    }
                }
            }
            if (lane == 0) {
                if (U.Vn) {
                    U.Nn[piece] |= grown;
                    U.Un[piece] |= fresh_blocks;
                }
                if (lost) {
                    // the wetting phase changed here: its tile is recomputed next step
                    const int nt1 = (G.b1 + kT1 - 1) / kT1;
                    U.wdirty[((c0 / kT0) * nt1 + c1 / kT1) * nt2 + tk] = 1;
                }
            }
        }
        __syncthreads(); // s_n and the list are written again
    }
    c2n = __reduce_add_sync(0xffffffffu, c2n);
    c1n = __reduce_add_sync(0xffffffffu, c1n);
    if (lane == 0 && c2n)
        atomicAdd(C.cnt2, (unsigned long long)c2n);
    if (lane == 0 && c1n)
        atomicAdd(C.cnt1, (unsigned long long)c1n);
    // the last block to finish: totals, and clean counters for the next radius
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(C.ticket, 1u) == gridDim.x - 1) {
        __threadfence();
        drain_totals(C, full);
        *C.kept = 0;
        C.xr[0] = C.xr[1] = 0;
        *C.ticket = 0u;
    }
}

int drain_same(const DrainCounts &C, cudaStream_t st)
{
    k_drain_same<<<1, 1, 0, st>>>(C);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

int drain_update_rows(uint8_t *mp, const unsigned *D, const int64_t *shape, ShrinkSel &w, const Boxes &B, GrowSel *g_nw,
                      const DrainCounts &C, int *err, cudaStream_t st, const int *orange, bool full)
{
    const BGrid G = bgrid_of(shape);
    UpdateSets U{};
    U.Vw = w.V;
    U.Mw = w.M;
    U.Pw = w.P;
    U.markw = w.mark;
    U.stamp = (uint8_t)w.stamp;
    U.wdirty = w.dirty;
    U.Tw = w.T;
    if (g_nw) {
        U.Vn = g_nw->V;
        U.Nn = g_nw->N;
        U.Un = g_nw->U;
        U.Mn = g_nw->M;
        U.Pn = g_nw->P;
    }
    const int ps__ = prof_begin("k_drain_update_rows", st);
    k_drain_update_rows<<<grid_for((row_pieces(G) + kUpdatePieces - 1) / kUpdatePieces * 256LL, 256, 152LL * 64), 256, 0,
                          st>>>(
        mp, D, U, G, (G.b2 + kT2 - 1) / kT2, B, C, err, orange, full ? 1 : 0, prof_units(kUnitsDrainUpdate));
    // per voxel visited: a bit of the dilation, of the wetting and of the
    // non-wetting phase
    prof_end_units(ps__, kUnitsDrainUpdate, 3.0 / 8.0, st);
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

// ---- binary labelling on blocks -----------------------------------------------
// connect_components (connected_components.py:32-62; cc3d numbers components
// 1..N in the order of their first voxel in C order) for an image with a
// single nonzero value: the block union-find gives the components, and the
// first voxel of each one is found and ranked without a per-voxel parent
// array.  The first voxel of a block is its lowest set mask bit (bit order
// x, y, z follows C order); the first voxel of a component lies in the
// component's first block plane (the plane of its root, the smallest block
// index), so only blocks of that plane compete for it.

__device__ __forceinline__ int block_first_voxel(const BGrid &G, int b, unsigned m)
{
    int c0, c1, c2;
    G.coords(b, c0, c1, c2);
    const int bit = __ffs(m) - 1;
    const int x = bit >> 2, y = (bit >> 1) & 1, z = bit & 1;
    return ((2 * c0 + x) * G.s1 + 2 * c1 + y) * G.s2 + 2 * c2 + z;
}

// Parents flattened to the roots, the roots listed (roots[0 .. *nroots), in no
// order) and F[root] lowered to the component's first voxel (unsigned, all ones
// before).  Four blocks per thread, so that their chains of dependent loads
// overlap: block by block this pass and a separate one for the first voxels
// took 2.0 ms at 1024^3.
__global__ void __launch_bounds__(256) k_blk_roots(int *__restrict__ P, const uint8_t *__restrict__ M, BGrid G,
                                                   unsigned *F, int *__restrict__ roots, int *nroots, int *err)
{
    const int nb = G.b0 * G.b1 * G.b2, plane = G.b1 * G.b2;
    const int lane = threadIdx.x & 31;
    constexpr int NB = 4;
    for (int base = blockIdx.x * blockDim.x * NB; base < nb; base += gridDim.x * blockDim.x * NB) {
        int b[NB], p[NB], g[NB];
        unsigned m[NB];
#pragma unroll
        for (int q = 0; q < NB; q++) {
            b[q] = base + q * blockDim.x + threadIdx.x;
            const bool in = b[q] < nb;
            p[q] = in ? ld(P + b[q]) : -1;
            m[q] = in ? M[b[q]] : 0u;
        }
#pragma unroll
        for (int q = 0; q < NB; q++)
            g[q] = p[q] >= 0 && p[q] != b[q] ? ld(P + p[q]) : p[q];
#pragma unroll
        for (int q = 0; q < NB; q++) {
            int r = p[q];
            if (r >= 0 && r != b[q]) {
                if (g[q] != r)
                    r = find_root(P, g[q], err);
                if (r != p[q])
                    P[b[q]] = r;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, r >= 0 && r == b[q]);
            if (bal) {
                int pos = 0;
                if (lane == 0)
                    pos = atomicAdd(nroots, __popc(bal));
                pos = __shfl_sync(0xffffffffu, pos, 0);
                if (r == b[q] && r >= 0)
                    roots[pos + __popc(bal & ((1u << lane) - 1u))] = r;
            }
            // the first voxel lies in the root's block plane
            if (r >= 0 && b[q] - r < plane) {
                int c0, c1, c2;
                G.coords(b[q], c0, c1, c2);
                if (r >= c0 * plane) {
                    const unsigned f = (unsigned)block_first_voxel(G, b[q], m[q]);
                    if (f < *(volatile unsigned *)(F + r))
                        atomicMin(F + r, f);
                }
            }
        }
    }
}

// bit f of `bits` set for every component's first voxel f
__global__ void k_blk_first_bits(const int *__restrict__ roots, const int *__restrict__ nroots,
                                 const unsigned *__restrict__ F, unsigned *bits)
{
    const int n = *nroots;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned f = F[roots[i]];
        atomicOr(bits + (f >> 5), 1u << (f & 31));
    }
}

// set bits per tile of 32 words (1024 voxels)
__global__ void k_bits_count(const unsigned *__restrict__ bits, long long nwords, int *cnt)
{
    const long long ntiles = (nwords + 31) / 32;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < ntiles;
         t += (long long)gridDim.x * blockDim.x) {
        int c = 0;
        const long long w1 = min(nwords, 32 * t + 32);
        for (long long w = 32 * t; w < w1; w++)
            c += __popc(bits[w]);
        cnt[t] = c;
    }
}

// root blocks: F[root] <- 1 + rank of its first voxel among all first voxels
__global__ void k_root_label(const int *__restrict__ roots, const int *__restrict__ nroots, unsigned *F,
                             const unsigned *__restrict__ bits, const int *__restrict__ offs)
{
    const int n = *nroots;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned f = F[roots[i]];
        const unsigned w = f >> 5;
        int r = offs[f >> 10] + __popc(bits[w] & ((1u << (f & 31)) - 1u));
        for (unsigned u = (f >> 10) * 32; u < w; u++)
            r += __popc(bits[u]);
        F[roots[i]] = (unsigned)r + 1u;
    }
}

// labels of every voxel: a block's label on its foreground voxels, 0 elsewhere
__global__ void k_blk_label_out(const int *__restrict__ P, const uint8_t *__restrict__ M, const unsigned *__restrict__ F,
                                BGrid G, uint64_t *__restrict__ labels, const uint64_t *__restrict__ lut)
{
    const int nb = G.b0 * G.b1 * G.b2;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        int c0, c1, c2;
        G.coords(b, c0, c1, c2);
        const unsigned m = M[b];
        uint64_t lab = m ? (uint64_t)F[P[b]] : 0;
        if (lut && lab)
            lab = lut[lab];
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
            for (int y = 0; y < 2; y++) {
                const int i = 2 * c0 + x, j = 2 * c1 + y;
                if (i >= G.s0 || j >= G.s1)
                    continue;
                uint64_t *row = labels + ((long long)i * G.s1 + j) * G.s2;
#pragma unroll
                for (int z = 0; z < 2; z++) {
                    const int k = 2 * c2 + z;
                    if (k < G.s2)
                        row[k] = ((m >> ((x * 2 + y) * 2 + z)) & 1u) ? lab : 0;
                }
            }
    }
}

// ... or computed from the block union-find: a voxel's label is its block's
// root's number when the voxel is foreground.
struct LabBlk {
    const int *P;
    const uint8_t *M;
    const unsigned *F;
    BGrid G;
    __device__ __forceinline__ uint64_t at(long long i, long long j, long long k) const
    {
        const int b = (int)(((i >> 1) * G.b1 + (j >> 1)) * G.b2 + (k >> 1));
        const int bit = (int)(((i & 1) * 2 + (j & 1)) * 2 + (k & 1));
        return ((M[b] >> bit) & 1u) ? (uint64_t)F[P[b]] : 0;
    }
};

// *single = 0 (and no labels) when the image holds two nonzero values, which
// the tile phase finds on the way: the caller then labels voxel by voxel.
static int cc_label_blocks(const uint8_t *img, uint64_t *labels, const int64_t *shape, const int32_t *bc,
                           const int32_t *pad, int64_t *count, int *single, cudaStream_t st)
{
    const BGrid G = bgrid_of(shape);
    const int nb = G.b0 * G.b1 * G.b2;
    const long long n = shape[0] * shape[1] * shape[2];
    const long long nwords = (n + 31) / 32, ntiles = (nwords + 31) / 32;
    // one allocation: parents, first voxels (then labels), roots, row words,
    // masks, first-voxel bits, their counts and offsets, scalars, scan scratch
    size_t tb = 0;
    PMG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, (int *)nullptr, (int *)nullptr, (int)ntiles + 1, st));
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t ib = up((size_t)nb * 4), cb = up((size_t)ntiles * 4 + 4);
    char *mem = nullptr;
    PMG_TRY(scratch_alloc((void **)&mem, 3 * ib + bcc_row_bytes(G) + up((size_t)nb) + up((size_t)nwords * 4) + 2 * cb +
                                            256 + tb,
                          st));
    char *p = mem;
    auto take = [&](size_t b) {
        char *q = p;
        p += b;
        return q;
    };
    int *P = (int *)take(ib);
    unsigned *F = (unsigned *)take(ib);
    int *roots = (int *)take(ib);
    unsigned *V = (unsigned *)take(bcc_row_bytes(G));
    uint8_t *M = (uint8_t *)take(up((size_t)nb));
    unsigned *bits = (unsigned *)take(up((size_t)nwords * 4));
    int *cnt = (int *)take(cb), *offs = (int *)take(cb);
    int *err = (int *)take(256), *nroots = err + 1;
    unsigned *range = (unsigned *)(err + 2); // OR, AND of the nonzero values
    void *tmp = p;
    auto run = [&]() -> int {
        PMG_CUDA(cudaMemsetAsync(err, 0, 3 * sizeof(int), st));
        PMG_CUDA(cudaMemsetAsync(range + 1, 0xff, sizeof(int), st));
        SrcImg src{img, -1};
        src.range = range;
        PMG_TRY(bcc_tile_phase(src, shape, P, M, V, st));
        unsigned h[2] = {0, 0};
        PMG_CUDA(cudaMemcpyAsync(h, range, sizeof(h), cudaMemcpyDeviceToHost, st));
        PMG_CUDA(cudaStreamSynchronize(st));
        *single = h[0] == 0 || h[0] == (h[1] & 0xffu);
        if (!*single)
            return PMG_OK;
        PMG_TRY(bcc_cross_phase(shape, bc, pad, false, P, M, V, err, st));
        PMG_CUDA(cudaMemsetAsync(F, 0xff, (size_t)nb * 4, st));
        PMG_CUDA(cudaMemsetAsync(bits, 0, (size_t)nwords * 4, st));
        {
            const int ps__ = prof_begin("k_blk_roots", st);
            k_blk_roots<<<grid_for((nb + 3) / 4, 256, 152LL * 32), 256, 0, st>>>(P, M, G, F, roots, nroots, err);
            k_blk_first_bits<<<152, 256, 0, st>>>(roots, nroots, F, bits);
            k_bits_count<<<grid_for(ntiles, 256, 152LL * 32), 256, 0, st>>>(bits, nwords, cnt);
            prof_end(ps__, (double)nb * 9 + (double)nwords * 4, st);
        }
        PMG_CHECK_LAUNCH();
        PMG_CUDA(cudaMemsetAsync(cnt + ntiles, 0, 4, st));
        size_t tb2 = tb;
        PMG_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb2, cnt, offs, (int)ntiles + 1, st));
        k_root_label<<<152, 256, 0, st>>>(roots, nroots, F, bits, offs);
        PMG_CHECK_LAUNCH();
        int total = 0;
        PMG_CUDA(cudaMemcpyAsync(&total, offs + ntiles, sizeof(int), cudaMemcpyDeviceToHost, st));
        PMG_TRY(read_err(err, st));
        // periodic seams: the relabelling table is built from the blocks' labels
        // on the seam slabs and folded into the one pass that writes the labels
        uint64_t *lut = nullptr;
        int64_t merged = total;
        if (any_periodic(bc))
            PMG_TRY(periodic_renumber(LabBlk{P, M, F, G}, labels, shape, bc, pad, total, &merged, st, &lut));
        {
            const int ps__ = prof_begin("k_blk_label_out", st);
            k_blk_label_out<<<grid_for(nb, 256, 152LL * 64), 256, 0, st>>>(P, M, F, G, labels, lut);
            prof_end(ps__, (double)n * 8 + (double)nb * 9, st);
            PMG_CHECK_LAUNCH();
        }
        if (lut)
            PMG_TRY(scratch_free(lut, st));
        *count = merged;
        return PMG_OK;
    };
    const int s = run();
    PMG_TRY(scratch_free(mem, st));
    return s;
}

int cc_label_u8(const uint8_t *img, uint64_t *labels, const int64_t *shape, const int32_t *bc, const int32_t *pad,
                int64_t *count, cudaStream_t st)
{
    int single = 0;
    PMG_TRY(cc_label_blocks(img, labels, shape, bc, pad, count, &single, st));
    return single ? PMG_OK : cc_label_t(img, labels, shape, bc, pad, count, st);
}

// Selection with caller-provided scratch: P (n int32), mark (n bytes rounded
// up to 4), err (one int, zeroed by the caller).  Does not synchronize.
int select_run(const uint8_t *img, void *out, int out_bytes, const int64_t *shape,
               const int32_t *bc, const int32_t *pad, const int64_t *inlet_box,
               const int64_t *outlet_box, int mode, int phase, int *P, uint8_t *mark, int *err,
               cudaStream_t st)
{
    const long long n = shape[0] * shape[1] * shape[2];
    PMG_CUDA(cudaMemsetAsync(mark, 0, ((size_t)n + 3) & ~(size_t)3, st));
    PMG_TRY(uf_build<uint8_t>(img, P, shape, bc, pad, true, err, st));
    Vol3 V{shape[0], shape[1], shape[2]};
    const int64_t *boxes[2] = {inlet_box, outlet_box};
    for (int w = 0; w < 2; w++) {
        const int64_t *bx = boxes[w];
        if (!bx || bx[0] < 0)
            continue;
        Box b;
        for (int d = 0; d < 3; d++) {
            b.lo[d] = bx[2 * d];
            b.hi[d] = bx[2 * d + 1];
            if (b.lo[d] < 0 || b.hi[d] > shape[d] || b.lo[d] > b.hi[d]) {
                set_error("connected-image selection: face box outside the volume");
                return PMG_EINVAL;
            }
        }
        if (b.size() > 0) {
            {
                const int ps__ = prof_begin("k_mark_face", st);
                k_mark_face<<<grid_for(b.size(), 256, 1LL << 30), 256, 0, st>>>(P, V, b, mark,
                                                                              (uint8_t)(1 << w));
                prof_end(ps__, (double)b.size() * 4, st);
            }
            PMG_CHECK_LAUNCH();
        }
    }
    if (out_bytes == 1)
        {
            const int ps__ = prof_begin("k_select", st);
            k_select<uint8_t><<<grid_for(n, 256, 1LL << 30), 256, 0, st>>>(img, P, mark, n, mode, phase,
                                                                        (uint8_t *)out);
            prof_end(ps__, (double)n * (5 + out_bytes), st);
        }
    else
        {
            const int ps__ = prof_begin("k_select", st);
            k_select<uint64_t><<<grid_for(n, 256, 1LL << 30), 256, 0, st>>>(img, P, mark, n, mode, phase,
                                                                         (uint64_t *)out);
            prof_end(ps__, (double)n * (5 + out_bytes), st);
        }
    PMG_CHECK_LAUNCH();
    return PMG_OK;
}

int check_err(int *err, cudaStream_t st) { return read_err(err, st); }

int check_volume(const int64_t *shape) { return check_vol(shape); }

} // namespace pmg

extern "C" int pmg_cc_select(const uint8_t *img, void *out, int32_t out_bytes,
                             const int64_t shape[3], const int32_t bc[6], const int32_t pad[6],
                             const int64_t inlet_box[6], const int64_t outlet_box[6], int32_t mode,
                             int32_t phase, void *stream)
{
    if (!img || !out || !shape || !bc || !pad) {
        set_error("pmg_cc_select: null argument");
        return PMG_EINVAL;
    }
    if (out_bytes != 1 && out_bytes != 8) {
        set_error("pmg_cc_select: output element size must be 1 or 8");
        return PMG_EINVAL;
    }
    const bool binary = (mode & PMG_SEL_BINARY) != 0;
    mode &= ~PMG_SEL_BINARY;
    if (mode < PMG_SEL_INLET || mode > PMG_SEL_ISOLATED) {
        set_error("pmg_cc_select: unknown mode %d", mode);
        return PMG_EINVAL;
    }
    PMG_TRY(check_geometry(shape, bc, pad));
    PMG_TRY(check_vol(shape));
    cudaStream_t st = as_stream(stream);
    const long long n = shape[0] * shape[1] * shape[2];
    int *P = nullptr, *err = nullptr;
    uint8_t *mark = nullptr;
    int s;
    if (phase >= 0 || binary) {
        const long long nb = ((shape[0] + 1) / 2) * ((shape[1] + 1) / 2) * ((shape[2] + 1) / 2);
        const size_t mb = ((size_t)nb + 255) & ~(size_t)255;
        PMG_TRY(scratch_alloc((void **)&P, (size_t)nb * 4, st));
        PMG_TRY(scratch_alloc((void **)&mark, 2 * mb, st));
        PMG_TRY(scratch_alloc((void **)&err, sizeof(int), st));
        PMG_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
        s = select_run_binary(img, out, out_bytes, shape, bc, pad, inlet_box, outlet_box, mode, phase >= 0 ? phase : -1,
                              P, mark, mark + mb, err, st, nullptr);
    } else {
        PMG_TRY(scratch_alloc((void **)&P, (size_t)n * 4, st));
        PMG_TRY(scratch_alloc((void **)&mark, ((size_t)n + 3) & ~(size_t)3, st));
        PMG_TRY(scratch_alloc((void **)&err, sizeof(int), st));
        PMG_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
        s = select_run(img, out, out_bytes, shape, bc, pad, inlet_box, outlet_box, mode, phase, P, mark, err, st);
    }
    if (s == PMG_OK)
        s = read_err(err, st);
    PMG_TRY(scratch_free(P, st));
    PMG_TRY(scratch_free(mark, st));
    PMG_TRY(scratch_free(err, st));
    return s;
}

// Testing aid: lower every union-find iteration cap (c_uf_cap) to `cap`
// (<= 0 restores the default bounds).
extern "C" int pmg_set_iteration_cap(int32_t cap)
{
    const int v = cap > 0 ? cap : INT_MAX;
    PMG_CUDA(cudaMemcpyToSymbol(c_uf_cap, &v, sizeof(int)));
    return PMG_OK;
}
