// Internal entry points shared between translation units (not part of the C ABI).
#pragma once

#include "pmg_common.cuh"

namespace pmg {

// rows (dilation): the seeds as row words (cc.cu: eight words per 32 2x2x2
// blocks of a row, bit c of word (x * 2 + y) * 2 + z for that voxel of block c;
// rows_bytes(shape)); img is then scratch of one byte per voxel, written only
// on the paths that need the seeds as bytes.  rows_out: the result as row words
// instead of bytes in out, which then is scratch too.
int morph_run(const uint8_t *img, uint8_t *out, const int64_t *shape, const int32_t *bc,
              const int32_t *pad, const int32_t *ext, const float *res, double radius, int cmp64,
              int dilate, uint8_t *E, float *A, float *B, cudaStream_t st, double thr_sq = -1.0,
              const unsigned long long *gate = nullptr, const int *xr = nullptr, int *orange = nullptr,
              const unsigned *rows = nullptr, unsigned *rows_out = nullptr);
size_t rows_bytes(const int64_t *shape);
int bytes_to_rows(const uint8_t *img, unsigned *V, const int64_t *shape, cudaStream_t st);
size_t morph_scratch_bytes(const int64_t *shape, const int32_t *bc, const int32_t *ext);
int erosion_edt_run(const uint8_t *img, float *D, const int64_t *shape, const int32_t *bc,
                    const int32_t *pad, const float *res, int unit_res, uint8_t *E, float *A,
                    cudaStream_t st);
int erosion_edt_ext_run(const uint8_t *img, float *D, const int64_t *shape, const int32_t *bc, const int32_t *pad,
                        const int32_t *ext, const float *res, int unit_res, uint8_t *E, float *A, int64_t *X,
                        int64_t *lo, cudaStream_t st);
int erosion_cap_run(const uint8_t *img, uint16_t *KC, const int64_t *shape, const int32_t *bc,
                    const int32_t *pad, int Tcap, uint16_t *KA, uint16_t *KB, int *flag, int *nonbinary,
                    cudaStream_t st);

int select_run(const uint8_t *img, void *out, int out_bytes, const int64_t *shape,
               const int32_t *bc, const int32_t *pad, const int64_t *inlet_box,
               const int64_t *outlet_box, int mode, int phase, int *P, uint8_t *mark, int *err,
               cudaStream_t st);
int select_run_binary(const uint8_t *img, void *out, int out_bytes, const int64_t *shape, const int32_t *bc,
                      const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box, int mode,
                      int fgval, int *P, uint8_t *M, uint8_t *mark, int *err, cudaStream_t st,
                      unsigned long long *kept = nullptr);
int select_run_erode(const uint16_t *E, int T, void *out, const int64_t *shape, const int32_t *bc,
                     const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box, int mode, int *P,
                     uint8_t *M, uint8_t *mark, int *err, cudaStream_t st, unsigned long long *kept = nullptr);

// Boxes of a drainage run: own voxels, inlet / outlet faces (lo0, hi0, lo1,
// hi1, lo2, hi2; lo0 < 0 for none), reservoir widths per face.
struct Boxes {
    int64_t own[6];
    int64_t inlet[6], outlet[6];
    int32_t rpad[6];
};

// Selection of a set that only grows from one call to the next (same shape,
// boundaries and boxes): the block union-find is kept and only blocks whose
// mask grew are united again.  Scratch of grow_sel_bytes(shape) bytes.
struct GrowSel {
    int *P = nullptr;
    uint8_t *M = nullptr;
    uint8_t *mark = nullptr;
    // row words; per 32 blocks of a row, the blocks that changed since the last
    // step's unions and those not yet connected to the inlet
    unsigned *V = nullptr;
    unsigned *N = nullptr;
    unsigned *U = nullptr;
    int2 *pairs = nullptr; // blocks to unite (npairs of them)
    int *npairs = nullptr;
    int stamp = 0; // of the last step's inlet marks
    bool built = false;
    // masks and words already brought up to date by the producer of the set
    // (the drainage update); the next step skips its mask pass
    bool pending = false;
    // blocks that grow at each step, known in advance (step_lists_build):
    // step k's blocks are ev[off[k] .. off[k + 1])
    int *ev = nullptr;
    int *off = nullptr;
};
// Per-step lists of the blocks of a step volume S (steps < nsteps; 255:
// never) that grow at that step, in one allocation *mem (freed by the caller).
int step_lists_build(GrowSel &g, const uint8_t *S, const int64_t *shape, int nsteps, void **mem, cudaStream_t st);
size_t grow_sel_bytes(const int64_t *shape);
void grow_sel_init(GrowSel &g, void *mem, const int64_t *shape);
int select_grow_binary(GrowSel &g, const uint8_t *img, int fgval, void *out, const int64_t *shape,
                       const int32_t *bc, const int32_t *pad, const int64_t *inlet_box, const int64_t *outlet_box,
                       int mode, int *err, cudaStream_t st, unsigned long long *kept = nullptr);
// A growing selection of a drainage radius up to its inlet stamps, no axis being
// periodic: the eroded space (step k of S when S is given, else E > T), the
// non-wetting phase (fgval in img).
int grow_marks_eroded(GrowSel &g, const uint8_t *S, int k, const uint16_t *E, int T, const int64_t *shape,
                      const int32_t *bc, const int32_t *pad, const int64_t *inlet_box, int *err, cudaStream_t st);
int grow_marks_phase(GrowSel &g, const uint8_t *img, int fgval, const int64_t *shape, const int32_t *bc,
                     const int32_t *pad, const int64_t *inlet_box, int *err, cudaStream_t st);
// The inlet selection of a constrained by b (when *b_count > 0) as row
// words; kept counts a's inlet-connected voxels, xr receives the x range of the
// output's set (kRangeBig encoding); both are zero before.
int grow_pair_select(GrowSel &a, GrowSel &b, const unsigned long long *b_count, unsigned *out, const int64_t *shape,
                     int *err, cudaStream_t st, unsigned long long *kept, int *xr);
// Selection of a set that only shrinks (the drainage's wetting phase): full
// block union-find every step, but tiles the producer did not flag keep their
// tile-local parents.  Scratch of shrink_sel_bytes(shape) bytes.
struct ShrinkSel {
    int *P = nullptr;
    unsigned *R = nullptr; // tile roots, one bit per block
    unsigned *T = nullptr; // blocks found cut off from the outlet, one bit per block
    uint8_t *M = nullptr;
    uint8_t *mark = nullptr;
    int *dirty = nullptr; // per tile: changed since the last step
    unsigned *V = nullptr; // row words of the masks
    int ntiles = 0;
    int stamp = 0; // of the last step's outlet marks
    bool built = false;
};
size_t shrink_sel_bytes(const int64_t *shape);
void shrink_sel_init(ShrinkSel &g, void *mem, const int64_t *shape);
int shrink_marks_binary(ShrinkSel &g, const uint8_t *img, int fgval, const int64_t *shape, const int32_t *bc,
                        const int32_t *pad, const int64_t *outlet_box, int *err, cudaStream_t st);
// The counts of a drainage curve (device): cnt2 and cnt1 of one update, their
// running totals tot and ones, the saturation numerator of the radius (sat), and
// what the next radius's selection counts into (kept, xr), cleared with them by
// the update's last block (ticket: its blocks done).
struct DrainCounts {
    unsigned long long *cnt2, *cnt1, *tot, *ones, *sat, *kept;
    int *xr;
    unsigned *ticket;
};
// The drainage update on row words: D the dilation (null: none), defined on
// the voxel x range orange (device, [lo, hi] in whole blocks, null:
// everything); full: every voxel and the reservoir slabs, the counts being all
// voxels of value 2 in the own box and the voxels newly 1; otherwise only the
// dilation's range, the counts being changes.  w's masks, words and tile flags
// are brought up to date, and g_nw's when given.
int drain_update_rows(uint8_t *mp, const unsigned *D, const int64_t *shape, ShrinkSel &w, const Boxes &B, GrowSel *g_nw,
                      const DrainCounts &C, int *err, cudaStream_t st, const int *orange, bool full);
int drain_same(const DrainCounts &C, cudaStream_t st); // a radius without change
int check_err(int *err, cudaStream_t st);
int check_volume(const int64_t *shape);

int update_buffer_run(void *img, int elem_bytes, const int64_t *shape, const int32_t *bc,
                      const int32_t *pad, cudaStream_t st);
int count_eq_async(const uint8_t *img, const int64_t *shape, const int64_t *box, uint8_t value,
                   unsigned long long *d_cnt, cudaStream_t st);

} // namespace pmg
