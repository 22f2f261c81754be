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
// costs B read and written once, which eight uses of each row repay for odd widths (200 000 rows of 8, 19 columns 68 -> 37
// us, 57 columns 81 -> 71; 20 000 rows of 24, 201 columns 61 -> 35; wider than 256 from 24 on: 200 000 of 8, 323 columns
// 430 and 445).  Even widths, whose rows of C are written in pairs, gain where their pairs leave lanes idle, from eleven uses on
// (300 000 even rows of 10 over 200 000, 50 columns 120 -> 97; 300 000 Zipf rows of 12, 130 columns 430 -> 373; 100 000 of
// 12, 150 columns 111 -> 100; with 59 of 64 lanes at work 33.9 and 35.5, with 31 of 32 87.6 and 87.3), of which 66 to 108
// columns have two pairs per lane already and need 24 (90 columns, 30 uses 82 -> 78; 98, 12 uses 31.9 and 35.1); up to 32 columns
// 30 from 16 on, eight whole vectors (500 000 of 14 142 -> 122), the others from 48 (22 columns, 150 uses 47 -> 41; 26, 30
// uses 59 and 60); the rest from 64 uses on (20 000 of 100, 510 columns 260 -> 240).  Below 64 MB of gather (250 for even widths: 50 columns, 220 MB 45.6 and 45.9) the launch costs more
// than it gives, and long rows of few columns leave too few lane groups when they are cut to vectors (20 000 of 100, 19
// columns 30 -> 35).
size_t padded_b_bytes(const csrspmm_b200_args* a);

void set_last_error(const char* fmt, ...);
const char* get_last_error();

}  // namespace csrspmm_b200
