// Compile-time tuning constants of the SpMM kernels.  Every value can be overridden on the
// compiler command line (-DCSRSPMM_TUNE_...=n) to build an experimental variant of the library;
// the defaults are the measured best on B200.
#pragma once

// SMs of the one GPU this library is for: what grids and thresholds are counted in
#ifndef CSRSPMM_TUNE_SMS
#define CSRSPMM_TUNE_SMS 148
#endif

// B-row loads kept in flight per lane, by number of column vectors per lane (NV) -- merge kernel
#ifndef CSRSPMM_TUNE_MERGE_U_NV1
#define CSRSPMM_TUNE_MERGE_U_NV1 5
#endif
#ifndef CSRSPMM_TUNE_MERGE_U_LONG
#define CSRSPMM_TUNE_MERGE_U_LONG 6
#endif
#ifndef CSRSPMM_TUNE_MERGE_U_NV2
#define CSRSPMM_TUNE_MERGE_U_NV2 4
#endif
#ifndef CSRSPMM_TUNE_MERGE_U_NV4
#define CSRSPMM_TUNE_MERGE_U_NV4 3
#endif
// ... and row kernel (row_unroll below)
#ifndef CSRSPMM_TUNE_ROW_U_NV1
#define CSRSPMM_TUNE_ROW_U_NV1 4
#endif
#ifndef CSRSPMM_TUNE_ROW_U_NV2
#define CSRSPMM_TUNE_ROW_U_NV2 2
#endif
#ifndef CSRSPMM_TUNE_ROW_U_NV4
#define CSRSPMM_TUNE_ROW_U_NV4 3
#endif
#ifndef CSRSPMM_TUNE_ROW_U_SHORT
#define CSRSPMM_TUNE_ROW_U_SHORT 6
#endif
// resident kernel: entries per CTA and row of B from which it is taken
#ifndef CSRSPMM_TUNE_RESIDENT_REUSE
#define CSRSPMM_TUNE_RESIDENT_REUSE 2
#endif
// mean row length up to which rows count as short
#ifndef CSRSPMM_TUNE_ROW_SHORT_MEAN
#define CSRSPMM_TUNE_ROW_SHORT_MEAN 48
#endif

// scheduled pieces (sliced_kernel.cuh): consecutive pieces per lane group
#ifndef CSRSPMM_TUNE_SLICED_PIECES_PER_GROUP
#define CSRSPMM_TUNE_SLICED_PIECES_PER_GROUP 1
#endif
// scheduled pieces: resident CTAs per SM asked of the compiler (caps the registers)
#ifndef CSRSPMM_TUNE_SLICED_MINB
#define CSRSPMM_TUNE_SLICED_MINB 2
#endif
// scheduled pieces load B with an evict_last policy (1) or plainly (0)
#ifndef CSRSPMM_TUNE_SLICED_EVICT_LAST
#define CSRSPMM_TUNE_SLICED_EVICT_LAST 0
#endif
// scheduled pieces write their slots with streaming stores (1) or plain ones (0): the slots are read
// back by another kernel and should not push the slab of B out of L2
#ifndef CSRSPMM_TUNE_SLICED_STREAM_SLOTS
#define CSRSPMM_TUNE_SLICED_STREAM_SLOTS 0
#endif

// Scheduled pieces (sliced_kernel.cuh): the gather is pipelined through shared memory, no gathered
// row is held in registers, so a lane can own more column vectors and a warp more pieces.  Per dense
// width class k: lanes per group G, vectors per lane NV, rows of B in flight per group D (a multiple
// of 4 and a power of two; G*NV*16*D*(256/G) = 64 KB of ring per CTA at every width).
#ifndef CSRSPMM_TUNE_P0_G
#define CSRSPMM_TUNE_P0_G 8
#endif
#ifndef CSRSPMM_TUNE_P0_NV
#define CSRSPMM_TUNE_P0_NV 1
#endif
#ifndef CSRSPMM_TUNE_P0_D
#define CSRSPMM_TUNE_P0_D 16
#endif
#ifndef CSRSPMM_TUNE_P1_G
#define CSRSPMM_TUNE_P1_G 8
#endif
#ifndef CSRSPMM_TUNE_P1_NV
#define CSRSPMM_TUNE_P1_NV 2
#endif
#ifndef CSRSPMM_TUNE_P1_D
#define CSRSPMM_TUNE_P1_D 8
#endif
#ifndef CSRSPMM_TUNE_P2_G
#define CSRSPMM_TUNE_P2_G 16
#endif
#ifndef CSRSPMM_TUNE_P2_NV
#define CSRSPMM_TUNE_P2_NV 2
#endif
#ifndef CSRSPMM_TUNE_P2_D
#define CSRSPMM_TUNE_P2_D 8
#endif
#ifndef CSRSPMM_TUNE_P3_G
#define CSRSPMM_TUNE_P3_G 32
#endif
#ifndef CSRSPMM_TUNE_P3_NV
#define CSRSPMM_TUNE_P3_NV 2
#endif
#ifndef CSRSPMM_TUNE_P3_D
#define CSRSPMM_TUNE_P3_D 8
#endif
#ifndef CSRSPMM_TUNE_P4_G
#define CSRSPMM_TUNE_P4_G 32
#endif
#ifndef CSRSPMM_TUNE_P4_NV
#define CSRSPMM_TUNE_P4_NV 4
#endif
#ifndef CSRSPMM_TUNE_P4_D
#define CSRSPMM_TUNE_P4_D 4
#endif

// merge-path kernel: walk a lane group's range with one loop (loads predicated on the batch length)
// instead of a loop of whole batches followed by the partial one
#ifndef CSRSPMM_TUNE_MERGE_ONE_LOOP
#define CSRSPMM_TUNE_MERGE_ONE_LOOP 0
#endif

// threads per CTA of the merge-path kernels (merge, bulk-copy): lane groups per CTA = this / G
// merge-path tile staging: global loads in flight per thread before the stores to shared memory
#ifndef CSRSPMM_TUNE_MERGE_STAGE_BATCH
#define CSRSPMM_TUNE_MERGE_STAGE_BATCH 6
#endif
#ifndef CSRSPMM_TUNE_MERGE_THREADS
#define CSRSPMM_TUNE_MERGE_THREADS 256
#endif

// L2 residency hints: rows of B loaded with an evict_last policy applied to this percentage of
// the lines, C written with streaming stores.  Both are OFF by default: on B200 neither helped
// (config 3, B = 2.1 x L2: 685 us without hints, 687-714 us with any combination of them).
#ifndef CSRSPMM_TUNE_B_EVICT_LAST_PCT
#define CSRSPMM_TUNE_B_EVICT_LAST_PCT 0
#endif
#ifndef CSRSPMM_TUNE_C_STREAMING
#define CSRSPMM_TUNE_C_STREAMING 0
#endif

// shared-memory row buffers per warp in the TMA kernel (bulk copies in flight per warp)
#ifndef CSRSPMM_TUNE_TMA_SLOTS
#define CSRSPMM_TUNE_TMA_SLOTS 4
#endif
// merge-path items per warp in the TMA kernel, and its requested CTAs per SM
#ifndef CSRSPMM_TUNE_TMA_TG
#define CSRSPMM_TUNE_TMA_TG 128
#endif
#ifndef CSRSPMM_TUNE_TMA_MINB
#define CSRSPMM_TUNE_TMA_MINB 2
#endif

// row kernel: how a group hands its G loaded (col, val) pairs to all its lanes: 1 = through a
// shared-memory slice (broadcast reads), 0 = lane to lane by shuffle
#ifndef CSRSPMM_TUNE_ROW_STAGE_SMEM
#define CSRSPMM_TUNE_ROW_STAGE_SMEM 1
#endif

// row kernel on short rows (mean of 64 non-zeros or fewer): at most this many CTAs per SM, each
// looping over rows, instead of one short-lived CTA per 128/G rows (0 = never)
#ifndef CSRSPMM_TUNE_ROW_PERSISTENT
#define CSRSPMM_TUNE_ROW_PERSISTENT 8
#endif

// ... for matrices whose mean row length is at most this
#ifndef CSRSPMM_TUNE_ROW_PERSISTENT_MAX_MEAN
#define CSRSPMM_TUNE_ROW_PERSISTENT_MAX_MEAN 64
#endif

// threads per CTA of the row kernel (128: 4 rows per CTA at G = 32; small CTAs keep the tail short
// when there are only a few thousand rows -- 4096 rows in 256-thread CTAs left a 15 % imbalance)
#ifndef CSRSPMM_TUNE_ROW_THREADS
#define CSRSPMM_TUNE_ROW_THREADS 128
#endif

// row kernel, few rows (fewer warps of work than 8 per SM): registers are plentiful and latency is
// everything, so many more loads are kept in flight per lane
#ifndef CSRSPMM_TUNE_ROW_ULOW_NV1
#define CSRSPMM_TUNE_ROW_ULOW_NV1 16
#endif
#ifndef CSRSPMM_TUNE_ROW_ULOW_NV2
#define CSRSPMM_TUNE_ROW_ULOW_NV2 8
#endif
#ifndef CSRSPMM_TUNE_ROW_ULOW_NV4
#define CSRSPMM_TUNE_ROW_ULOW_NV4 4
#endif

// minimum resident CTAs per SM requested from the compiler (caps registers per thread)
#ifndef CSRSPMM_TUNE_MERGE_MINB_NV1
#define CSRSPMM_TUNE_MERGE_MINB_NV1 4
#endif
#ifndef CSRSPMM_TUNE_MERGE_MINB_NV2
#define CSRSPMM_TUNE_MERGE_MINB_NV2 3
#endif
#ifndef CSRSPMM_TUNE_MERGE_MINB_NV4
#define CSRSPMM_TUNE_MERGE_MINB_NV4 2
#endif
#ifndef CSRSPMM_TUNE_ROW_MINB_NV1
#define CSRSPMM_TUNE_ROW_MINB_NV1 8
#endif
#ifndef CSRSPMM_TUNE_ROW_MINB_NV2
#define CSRSPMM_TUNE_ROW_MINB_NV2 8
#endif
#ifndef CSRSPMM_TUNE_ROW_MINB_NV4
#define CSRSPMM_TUNE_ROW_MINB_NV4 4
#endif

// lane-group shapes by dense width class k (column vectors per row <= 8, 16, 32, 64, more):
// lanes per group G, vectors per lane NV, merge-path items per group TG.  TG = 192 against 128:
// fewer, longer-lived CTAs (one search, one staging round and one carry row each) -- config 3
// 686 -> 654 us, the same matrix at Nd = 128 1361 -> 1285 us, config 5 at a quarter of its rows
// 10.26 -> 10.04 ms; 224-384 gained nothing more at G = 32, whose walks wait for HBM, and TG = 256 at G = 16 no longer
// fits the 48 KB of static shared memory.  G = 8: 96, the same 3072 items per CTA as G = 16 (64 before): 32 columns, 1 M
// Zipf rows of 12 244 -> 226 us, 400 000 of 6 76 -> 72, 2 M of 4 268 -> 251, 500 000 even rows of 10 94.7 -> 90.7; 20 columns,
// 300 000 of 30 140 -> 128
#ifndef CSRSPMM_TUNE_S0_G
#define CSRSPMM_TUNE_S0_G 8
#endif
#ifndef CSRSPMM_TUNE_S0_NV
#define CSRSPMM_TUNE_S0_NV 1
#endif
#ifndef CSRSPMM_TUNE_S0_TG
#define CSRSPMM_TUNE_S0_TG 96
#endif
#ifndef CSRSPMM_TUNE_S1_G
#define CSRSPMM_TUNE_S1_G 16
#endif
#ifndef CSRSPMM_TUNE_S1_NV
#define CSRSPMM_TUNE_S1_NV 1
#endif
#ifndef CSRSPMM_TUNE_S1_TG
#define CSRSPMM_TUNE_S1_TG 192
#endif
#ifndef CSRSPMM_TUNE_S2_G
#define CSRSPMM_TUNE_S2_G 32
#endif
#ifndef CSRSPMM_TUNE_S2_NV
#define CSRSPMM_TUNE_S2_NV 1
#endif
#ifndef CSRSPMM_TUNE_S2_TG
#define CSRSPMM_TUNE_S2_TG 192
#endif
#ifndef CSRSPMM_TUNE_S3_G
#define CSRSPMM_TUNE_S3_G 32
#endif
#ifndef CSRSPMM_TUNE_S3_NV
#define CSRSPMM_TUNE_S3_NV 2
#endif
#ifndef CSRSPMM_TUNE_S3_TG
#define CSRSPMM_TUNE_S3_TG 192
#endif
#ifndef CSRSPMM_TUNE_S4_G
#define CSRSPMM_TUNE_S4_G 32
#endif
#ifndef CSRSPMM_TUNE_S4_NV
#define CSRSPMM_TUNE_S4_NV 4
#endif
#ifndef CSRSPMM_TUNE_S4_TG
#define CSRSPMM_TUNE_S4_TG 192
#endif

namespace csrspmm_b200 {

constexpr int kSms = CSRSPMM_TUNE_SMS;

// merge kernel: lane groups take no fewer items than this, and tiles of up to TG_SMALL items per group run the
// build that has shared memory for just those (more of it left to L1)
#ifndef CSRSPMM_TUNE_MERGE_TG_LEAST
#define CSRSPMM_TUNE_MERGE_TG_LEAST 16
#endif
#ifndef CSRSPMM_TUNE_MERGE_TG_SMALL
#define CSRSPMM_TUNE_MERGE_TG_SMALL 64
#endif

struct ShapeDesc {
    int G, NV, TG;
};
// Merge-path kernel on very narrow dense operands (1, 2 or 4 column vectors: Nd <= 4, 8, 16 with the
// 16-byte layout): a lane group of eight would leave seven, six or four of its lanes without a column,
// so the groups shrink to 1, 2 or 4 lanes -- at G = 1 every lane walks its own run of non-zeros
// (lanes over non-zeros instead of lanes over columns) and the rows cut between lanes are summed in
// lane order through shared memory like any other split row.  3072 merge-path items per CTA as for
// the wider shapes.
#ifndef CSRSPMM_TUNE_MERGE_NARROW
#define CSRSPMM_TUNE_MERGE_NARROW 1
#endif
constexpr int kNumNarrowShapes = 3;
constexpr ShapeDesc kNarrowShapes[kNumNarrowShapes] = {{1, 1, 12}, {2, 1, 24}, {4, 1, 48}};
struct PieceShapeDesc {
    int G, NV, D;
};
constexpr PieceShapeDesc kPieceShapes[5] = {
    {CSRSPMM_TUNE_P0_G, CSRSPMM_TUNE_P0_NV, CSRSPMM_TUNE_P0_D}, {CSRSPMM_TUNE_P1_G, CSRSPMM_TUNE_P1_NV, CSRSPMM_TUNE_P1_D},
    {CSRSPMM_TUNE_P2_G, CSRSPMM_TUNE_P2_NV, CSRSPMM_TUNE_P2_D}, {CSRSPMM_TUNE_P3_G, CSRSPMM_TUNE_P3_NV, CSRSPMM_TUNE_P3_D},
    {CSRSPMM_TUNE_P4_G, CSRSPMM_TUNE_P4_NV, CSRSPMM_TUNE_P4_D}};
constexpr int kNumShapes = 5;
constexpr ShapeDesc kShapes[kNumShapes] = {
    {CSRSPMM_TUNE_S0_G, CSRSPMM_TUNE_S0_NV, CSRSPMM_TUNE_S0_TG}, {CSRSPMM_TUNE_S1_G, CSRSPMM_TUNE_S1_NV, CSRSPMM_TUNE_S1_TG},
    {CSRSPMM_TUNE_S2_G, CSRSPMM_TUNE_S2_NV, CSRSPMM_TUNE_S2_TG}, {CSRSPMM_TUNE_S3_G, CSRSPMM_TUNE_S3_NV, CSRSPMM_TUNE_S3_TG},
    {CSRSPMM_TUNE_S4_G, CSRSPMM_TUNE_S4_NV, CSRSPMM_TUNE_S4_TG}};

constexpr int merge_unroll(int nv) { return nv == 1 ? CSRSPMM_TUNE_MERGE_U_NV1 : (nv == 2 ? CSRSPMM_TUNE_MERGE_U_NV2 : CSRSPMM_TUNE_MERGE_U_NV4); }
constexpr int row_unroll(int nv) { return nv == 1 ? CSRSPMM_TUNE_ROW_U_NV1 : (nv == 2 ? CSRSPMM_TUNE_ROW_U_NV2 : CSRSPMM_TUNE_ROW_U_NV4); }
constexpr int row_unroll_low(int nv) { return nv == 1 ? CSRSPMM_TUNE_ROW_ULOW_NV1 : (nv == 2 ? CSRSPMM_TUNE_ROW_ULOW_NV2 : CSRSPMM_TUNE_ROW_ULOW_NV4); }
// vector width 2 (rows on 8-byte boundaries): as many loads in flight as the same registers hold; width 1: eight
#ifndef CSRSPMM_TUNE_PAIR_U_NV1
#define CSRSPMM_TUNE_PAIR_U_NV1 6
#endif
#ifndef CSRSPMM_TUNE_PAIR_U_WIDE
#define CSRSPMM_TUNE_PAIR_U_WIDE 4
#endif
constexpr int merge_unroll(int vw, int nv)
{
    return vw == 4 ? merge_unroll(nv) : vw == 1 ? 8 : nv == 1 ? CSRSPMM_TUNE_PAIR_U_NV1 : CSRSPMM_TUNE_PAIR_U_WIDE;
}
// Row kernel: six loads in flight for short rows of one vector per lane where the registers last (64 columns, rows of 16:
// 65 536 of them 30.6 -> 24.4 us, 16 384 10.3 -> 8.6; 32 columns, rows of 8 15.2 -> 12.5), four where they do not (a column
// guard; 128 columns: 12.0 us with four, 12.6 with six) and for long rows, whose chunks of G entries are then whole batches
// (30 columns, rows of 100: 25.9 us with four, 31.6 with six).  Three with four vectors per lane (8192 rows, 4096
// columns: 239 us with four, 212 with three, 234 with two).
constexpr int row_unroll(int vw, int g, int nv, bool full, bool short_rows)
{
    if (vw == 1) return 8;
    if (nv > 1) return vw == 4 ? row_unroll(nv) : CSRSPMM_TUNE_PAIR_U_WIDE;
    return short_rows && (vw == 2 || (full && g <= 16)) ? CSRSPMM_TUNE_ROW_U_SHORT : CSRSPMM_TUNE_ROW_U_NV1;
}

// Row kernel on long rows (a mean above CSRSPMM_TUNE_ROW_SHORT_MEAN), where the grid is a wave or two and a wave lasts as long as
// a row: more rows of B in flight and fewer CTAs per SM where the grid does not fill them, or would leave a nearly empty wave behind.
// Grids in CTAs per SM.  Every line was measured on both sides: 870 products, rows of 49 to 900 entries, B of 0.1 to 240 MB, a quarter of
// them packed (the long grids' time over this build's, mean and range).  "Full": every lane at work (32, 64, 128, 256 columns).
//   1  one vector per lane, up to 4: 16 or 32 lanes 1.12, 0.99-1.25; eight, full 1.19, 1.05-1.31 (not full 1.00, 0.91-1.04)
//      two, up to 4: 1.36, 1.19-1.63; 8 to 10: 1.06, 0.95-1.18
//      four, 4 to 6: 1.16, 1.07-1.31; 8 to 9: 1.12, 0.98-1.21
//   2  8 to 12: eight lanes 1.09, 1.00-1.37; sixteen, full 1.12, 1.01-1.21, not full 1.00, 0.94-1.13; 32, full 1.09, 0.93-1.23, not full 1.03,
//      0.94-1.19
//      up to 6: eight lanes 1.04, 0.97-1.20; sixteen, full 1.07, 0.97-1.12 (not full 0.96, 0.94-0.98: 48 columns, rows of 115 15.8 and
//      16.5 us)
//   3  6 to 7: eight or sixteen lanes, full 1.11, 1.08-1.14 (32 columns, rows of 595 94.2 and 82.3; not full 0.91, 0.85-0.96: 24 columns,
//      rows of 323 55.9 and 62.1)
// Elsewhere each of them loses (6 to 8, build 2: 0.69, 0.58-0.85).
struct RowBuild {
    int U, MINB;
};
constexpr RowBuild row_build(int nv, int k)
{
    if (nv == 1) return k == 1 ? RowBuild{16, 4} : (k == 2 ? RowBuild{8, 6} : RowBuild{8, 7});
    return nv == 2 ? RowBuild{6, 4} : RowBuild{4, 3};
}
// 0: the long grids' build
constexpr int row_build_for(int g, int nv, bool full, long long grid)
{
    if (nv == 1) {
        if (grid <= kSms * 4) return g >= 16 || full ? 1 : 2;
        if (g <= 16 && grid <= kSms * 6) return full || g == 8 ? 2 : 0;
        if (g <= 16 && grid <= kSms * 7) return full ? 3 : 0;
        return grid > kSms * 8 && grid <= kSms * 12 ? 2 : 0;
    }
    if (nv == 2) return grid <= kSms * 4 || (grid > kSms * 8 && grid <= kSms * 10) ? 1 : 0;
    return (grid > kSms * 4 && grid <= kSms * 6) || (grid > kSms * 8 && grid <= kSms * 9) ? 1 : 0;
}
// What row_build_for can answer.
constexpr bool row_build_used(int g, int nv, bool full, int k)
{
    if (nv > 1) return k == 1;
    return k == 1 ? g >= 16 || full : k == 2 || (g <= 16 && full);
}

constexpr int row_min_blocks(int nv) { return nv == 1 ? CSRSPMM_TUNE_ROW_MINB_NV1 : (nv == 2 ? CSRSPMM_TUNE_ROW_MINB_NV2 : CSRSPMM_TUNE_ROW_MINB_NV4); }
constexpr int merge_min_blocks(int nv) { return nv == 1 ? CSRSPMM_TUNE_MERGE_MINB_NV1 : (nv == 2 ? CSRSPMM_TUNE_MERGE_MINB_NV2 : CSRSPMM_TUNE_MERGE_MINB_NV4); }

}  // namespace csrspmm_b200
