// Host-only launch planning for the SpMM entry point: which kernel, which lane-group shape,
// how many tiles, how much scratch.  Pure C++ (no CUDA call), so it can be unit-tested on a
// machine without a GPU.  Replaces the fixed geometry of the reference's launchers
// (src/host/spmm_launcher.cu:17-19, 63-66, 112-120) and the stub auto-selection of
// src/csrspmm.cpp:34-40.
#pragma once

#include <cstddef>
#include <cstdint>

#include "../kernels/tuning.h"
#include "csrspmm_b200.h"

namespace csrspmm_b200 {

struct Plan {
    int kernel = CSRSPMM_B200_KERNEL_ROW;  // resolved, never AUTO
    int shape = 0;                         // index into kShapes (tuning.h)
    bool low_occupancy = false;            // row kernel: fewer than 8 warps of rows per SM
    bool any_count = false;                // whole-row mapping of more than kWholeRowEntries entries: the panel kernel, one pass
    int resident = 0;                      // whole-row mapping by the resident kernel: lanes per group (16, 32), else 0
    int c_ragged = 0;                      // kPlanPadded: the last vector of a row of C is partly beyond it (SpmmParams::c_ragged)
    bool rows_even = false;                // AUTO: the longest row is known to be close to the mean
    bool short_rows = false;               // row kernel: mean of CSRSPMM_TUNE_ROW_SHORT_MEAN entries or fewer
    int row_build = 0;                     // row kernel, long rows, vector width 4: row_build_for()
    bool full = false;                     // one pass covers the row exactly: G*NV == ncolv
    bool row_aligned = false;              // merge kernel: tiles cut at row starts, no carries and no fix-up
    bool small_tile = false;               // merge kernel: the build with shared memory for small tiles
    int narrow = 0;                        // merge kernel: 1 + index into kNarrowShapes when the dense operand has at
                                           // most four column vectors (lane groups of 1, 2 or 4 lanes), else 0
    bool fills_chip = false;               // the grid takes every CTA slot of the chip at least once
    int G = 8, NV = 1, VW = 4;             // lanes per group, vectors per lane, vector width
    int ncolv = 0;                         // ceil(Nd / VW)
    int tg = 0;                            // merge-path items per lane group (split kernels)
    int tile = 0;                          // merge-path items per CTA (split kernels)
    long long num_items = 0;               // M + nnz
    long long num_tiles = 0;               // CTAs of the split kernels
    long long grid = 0;                    // CTAs of the main kernel
    long long carry_ld = 0;                // floats per carry row
    size_t carry_row_bytes = 0;            // 256-byte aligned
    size_t workspace_bytes = 0;            // carry_row_bytes + carry values
    size_t dynamic_smem = 0;               // TMA kernel only: 8 warps x ring_stride
    size_t tma_slot_bytes = 0;             // TMA kernel only: one row of B rounded up to 128 bytes
};

// Entries up to which the row and resident kernels' int positions, which run up to 63 beyond the last one, do not wrap.  The
// panel kernel counts in unsigned and gives the same result, so it takes the few sizes above.
constexpr int64_t kWholeRowEntries = 0x7fffffffLL - 64;

// Checks the argument block (sizes, enums, pointers) without touching memory.
int check_args(const csrspmm_b200_args* a, bool need_pointers);

// True when every row of B and C, and both base pointers, allow 16-byte vector access.
bool vector_layout_ok(const csrspmm_b200_args* a);

// Resolves AUTO (and the CSRSPMM_FORCE_KERNEL override) and fills the launch geometry.
// Returns CSRSPMM_B200_OK or an error status.
constexpr unsigned kPlanNoNarrow = 1;  // no lane groups of fewer than eight lanes
constexpr unsigned kPlanCoarse = 2;    // no tiles smaller than 64 items per lane group: fewer carry rows
constexpr unsigned kPlanPadded = 8;    // for a copy of B padded to whole vectors (padded_b_bytes)
constexpr unsigned kPlanNoPairs = 4;   // vector widths 4 and 1 only
int make_plan(const csrspmm_b200_args* a, Plan* plan, unsigned flags = 0);

// What csrspmm_b200_spmm runs without a schedule: the plan for a padded copy of B (plan->c_ragged) when that pays and
// args.workspace has room for it behind the carries, at padded_b_offset(); else the plan for B as it is.
int product_plan(const csrspmm_b200_args* a, Plan* plan);
inline size_t padded_b_offset(const Plan& plan) { return (plan.workspace_bytes + 255) / 256 * 256; }

// Workspace of the split kernels whatever the plan: what csrspmm_b200_workspace_bytes reports (the larger of the MERGE
// and TMA needs), and enough for any contiguous block of the matrix's rows multiplied on its own.
size_t worst_case_workspace(const csrspmm_b200_args* a);

// Scratch for a copy of B with rows padded to whole 16-byte vectors, or 0 where the product does without.  Rows of
// 57 or 150 columns start on any 4 or 8 bytes, and gathered one or two floats per lane they come at half the rate; a copy
// costs B read and written once, and a launch.
// Odd widths: from eight uses of each row of B on (200 000 rows of 8, 19 columns 68 -> 37 us, 57 columns 81 -> 71; 20 000 rows of 24, 201
// columns 61 -> 35; wider than 256 from 24 on: 200 000 of 8, 323 columns 430 and 445) and 64 MB of gather; long rows of few columns leave
// too few lane groups when they are cut to vectors (20 000 of 100, 19 columns 30 -> 35).  Over 360 products of both sides 1.33.
// Even widths, whose rows of C are written in pairs.  Both sides measured on 1270 products, 18 to 510 columns, 6 to 250 uses, 0.2 to 5
// GB of gather, even and Zipf rows (time without the copy over time with it; mean, range, and the share that loses 2 % and more):
//   up to 32 columns, 48 uses (30 columns, eight whole vectors: 16): 1.11, 0.87-1.52, 6 %.  Not the rows of over 64 entries that fill one wave of
//     eight-lane groups and leave half of the next one empty (19 010 of 370, 22 columns 81 and 102)
//   pairs that leave lanes of a group idle: 34 to 54 columns, 24 uses 1.15, 0.87-1.51, 2 %, and rows known to be even from 11 uses on (11 to
//     24: even 1.11, 0.94-1.26, 2 of 12: 300 000 of 10 over 200 000, 50 columns 120 -> 97; uneven 0.99, 0.92-1.11, 7 of 20: 50 columns,
//     15 uses 761 and 825); 66 to 108, 24 uses 1.11, 0.92-1.36, 6 %; 130 to 216, 11 uses 1.17, 0.90-1.54, 6 %
//   other widths from 96 on, 64 uses: up to 256 1.07, 0.89-1.30, 15 %, beyond 1.16, 0.85-1.52, 5 %
// Below 250 MB of gather the launch costs more than it gives (50 columns, 220 MB 45.6 and 45.9).
size_t padded_b_bytes(const csrspmm_b200_args* a);

void set_last_error(const char* fmt, ...);
const char* get_last_error();

}  // namespace csrspmm_b200
