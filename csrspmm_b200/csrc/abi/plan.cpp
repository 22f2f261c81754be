// Host-only launch planning (see plan.h).
#include "plan.h"

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace csrspmm_b200 {

namespace {
thread_local char g_last_error[512] = "";

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
}  // namespace

void set_last_error(const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
    va_end(ap);
}

const char* get_last_error() { return g_last_error; }

int check_args(const csrspmm_b200_args* a, bool need_pointers)
{
    if (a == nullptr) {
        set_last_error("args is null");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->struct_size != sizeof(csrspmm_b200_args)) {
        set_last_error("args.struct_size is %u, this library expects %zu", a->struct_size,
                       sizeof(csrspmm_b200_args));
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->M < 0 || a->Kd < 0 || a->Nd < 0 || a->nnz < 0 || a->nnz > 0x7fffffffLL) {
        set_last_error("negative or oversized dimension (M=%d Kd=%d Nd=%d nnz=%lld)", a->M, a->Kd,
                       a->Nd, (long long)a->nnz);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->row_ptr_base < 0) {
        set_last_error("negative row_ptr_base %d", a->row_ptr_base);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->row_ptr_base != 0 && a->value_format == CSRSPMM_B200_VALUES_E2M1 && (a->row_ptr_base & 1)) {
        set_last_error("row_ptr_base must be even for packed e2m1 values (two codes per byte)");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->nnz > 0 && a->Kd == 0) {
        set_last_error("nnz > 0 with Kd == 0");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->ldb >= (1LL << 30) || a->ldc >= (1LL << 30)) {
        set_last_error("leading dimension of 2^30 elements or more (ldb=%lld ldc=%lld)", (long long)a->ldb,
                       (long long)a->ldc);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->ldb < a->Nd || a->ldc < a->Nd) {
        set_last_error("leading dimension smaller than Nd (ldb=%lld ldc=%lld Nd=%d)",
                       (long long)a->ldb, (long long)a->ldc, a->Nd);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->value_format != CSRSPMM_B200_VALUES_F32 && a->value_format != CSRSPMM_B200_VALUES_E2M1) {
        set_last_error("unknown value_format %d", a->value_format);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->entry < CSRSPMM_B200_ENTRY_NAIVE || a->entry > CSRSPMM_B200_ENTRY_WARP_PER_ROW_SMEM_FP4) {
        set_last_error("unknown entry %d", a->entry);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (a->kernel < CSRSPMM_B200_KERNEL_AUTO || a->kernel > CSRSPMM_B200_KERNEL_TMA) {
        set_last_error("unknown kernel %d", a->kernel);
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (need_pointers && a->M > 0 && a->Nd > 0) {
        if (a->row_ptr == nullptr || a->C == nullptr ||
            (a->nnz > 0 && (a->col_idx == nullptr || a->values == nullptr || a->B == nullptr))) {
            set_last_error("null matrix pointer");
            return CSRSPMM_B200_ERR_BAD_ARG;
        }
    }
    return CSRSPMM_B200_OK;
}

bool vector_layout_ok(const csrspmm_b200_args* a)
{
    return a->Nd % 4 == 0 && a->ldb % 4 == 0 && a->ldc % 4 == 0 &&
           (reinterpret_cast<uintptr_t>(a->B) & 15u) == 0 &&
           (reinterpret_cast<uintptr_t>(a->C) & 15u) == 0;
}

static bool pair_layout_ok(const csrspmm_b200_args* a)
{
    return a->Nd % 2 == 0 && a->ldb % 2 == 0 && a->ldc % 2 == 0 && (reinterpret_cast<uintptr_t>(a->B) & 7u) == 0 &&
           (reinterpret_cast<uintptr_t>(a->C) & 7u) == 0;
}

static int shape_for(int ncolv)
{
    if (ncolv <= 8) return 0;
    if (ncolv <= 16) return 1;
    if (ncolv <= 32) return 2;
    if (ncolv <= 64) return 3;
    return 4;
}

static bool tma_can_run(const csrspmm_b200_args* a)
{
    return vector_layout_ok(a) && a->Nd >= 4 && a->Nd <= 512;
}

static int forced_kernel_from_env()
{
    const char* e = std::getenv("CSRSPMM_FORCE_KERNEL");
    if (e == nullptr || *e == 0) return CSRSPMM_B200_KERNEL_AUTO;
    if (!std::strcmp(e, "row")) return CSRSPMM_B200_KERNEL_ROW;
    if (!std::strcmp(e, "merge")) return CSRSPMM_B200_KERNEL_MERGE;
    if (!std::strcmp(e, "tma")) return CSRSPMM_B200_KERNEL_TMA;
    return CSRSPMM_B200_KERNEL_AUTO;
}

static void fill_split_geometry(const csrspmm_b200_args* a, Plan* plan, int groups, int tg)
{
    plan->tg = tg;
    plan->tile = groups * tg;
    plan->num_items = (long long)a->M + a->nnz;
    plan->num_tiles = (plan->num_items + plan->tile - 1) / plan->tile;
    plan->grid = plan->num_tiles;
    plan->carry_ld = ((long long)a->Nd + 3) / 4 * 4;
    plan->carry_row_bytes = align_up((size_t)plan->num_tiles * sizeof(int32_t), 256);
    plan->workspace_bytes =
        plan->carry_row_bytes + (size_t)plan->num_tiles * (size_t)plan->carry_ld * sizeof(float);
}

// Items per lane group of the merge kernel: up to three waves of CTAs get tiles of one size that fill the waves;
// longer grids take the largest tile (most).  A tile of fixed size left 1.1 M items with 363 CTAs for 592 slots, and
// problems of a few ten thousand items with 64-item walks on a few CTAs: 65 536 rows of 16, 64 columns 32.0 -> 27.9 us,
// 16 384 rows of 16, 256 columns 31.7 -> 23.3, 16 384 rows of 4, 64 columns 13.6 -> 10.4, 1024 rows 11.7 -> 7.7.  Beyond
// three waves equal tiles gain nothing and their CTAs march in step (1 M rows of 16: 618 us against 600).  Not below
// `least`: a CTA's search and staging cost as much as a walk of some 16 items.
static int merge_items_per_group(long long num_items, int groups, int ctas_per_sm, int most, int least)
{
    const long long wave = (long long)kSms * ctas_per_sm * groups;
    const long long waves = (num_items + wave * most - 1) / (wave * most);
    if (waves > 3) return most;
    const long long tg = waves > 0 ? (num_items + wave * waves - 1) / (wave * waves) : 1;
    return (int)(tg < least ? least : (tg > most ? most : tg));
}

// Whether the merge kernel can cut its tiles at row starts: a tile and the longest row behind it have to fit the
// shared memory of the largest tile, and the grid to be short enough for the fix-up kernel to be worth saving.
static bool rows_fit_tiles(const csrspmm_b200_args* a, const Plan& plan, int groups, int most)
{
    return a->max_row_nnz > 0 && plan.tg < most && (long long)plan.tile + a->max_row_nnz + 1 <= (long long)groups * most;
}

// Lanes per group of the resident kernel for this product, 0 when the row kernel is the better one.  A panel of B has to
// fit shared memory (4 floats per lane and row of B) and to be used often enough to pay for being loaded; rows have to
// be long enough to hide the next row's bounds and entries (4096 x 128 times 4096 columns, rows of 1.3: 23.8 us against
// 21.1; of 6.4: 32.1 against 38.8).  Widths that the row kernel covers exactly in one pass it does well itself, helped by L1
// (6000 x 800 times 512 columns, rows of 100: 52 us against 66; 60 000 x 400 times 128, rows of 20: 35 against 30).
static int resident_lanes(const csrspmm_b200_args* a, const Plan& plan)
{
    if (plan.VW != 4 || a->Kd <= 0 || a->max_row_nnz <= 0 || a->nnz < 4LL * a->M) return 0;
    const int lanes = a->Kd * 512LL <= 200 * 1024 && plan.ncolv > 16 ? 32 : (a->Kd * 256LL <= 200 * 1024 ? 16 : 0);
    if (lanes == 0 || plan.ncolv < lanes || (plan.full && lanes == 16)) return 0;
    const long long panels = (plan.ncolv + lanes - 1) / lanes;
    const long long reuse = plan.full ? 16 : CSRSPMM_TUNE_RESIDENT_REUSE;  // entries per CTA and row of B
    return a->nnz * panels >= reuse * (long long)kSms * a->Kd ? lanes : 0;
}

// Whether a whole-row product would be a chain of its longest rows' entries on a chip that is mostly idle: few rows, long
// ones, and lane groups that share a warp, where the merge kernel cuts rows among all SMs.  512 rows of 200: 16 columns
// 25.3 us whole and 9.1 cut, 64 12.4 and 7.3, 512 22.6 and 16.1; 8192 rows of 200: 32 columns 34.7 and 22.5, 64 31.4 and 27.8;
// 18 000 of 100, 32 columns 23.4 and 24.5.  Widths that are no multiple of four lose earlier: their gather costs the
// merge kernel more (50 columns, rows of 200: 16.7 and 7.6 with 512 rows, 36.0 and 40.4 with 8192).
static bool rows_are_chains(long long M, double mean, const Plan& plan)
{
    const ShapeDesc& s = kShapes[shape_for(plan.ncolv)];
    if (plan.VW == 4) return s.G == 32 ? M < 592 && mean >= 200.0 : M <= 12000 && mean >= (s.G == 8 ? 64.0 : 150.0);
    return s.G == 32 ? M < 592 && mean >= (s.NV == 1 ? 80.0 : 200.0) : M <= 2400 && mean >= 80.0;
}

// Whether the longest row is known and close to the mean.
static bool rows_known_even(const csrspmm_b200_args* a, double mean)
{
    return a->max_row_nnz > 0 && (double)a->max_row_nnz <= (mean * 4.0 > 64.0 ? mean * 4.0 : 64.0);
}

int make_plan(const csrspmm_b200_args* a, Plan* plan, unsigned flags)
{
    const bool coarse = (flags & kPlanCoarse) != 0;
    int st = check_args(a, false);
    if (st != CSRSPMM_B200_OK) return st;
    *plan = Plan();
    const bool vec = vector_layout_ok(a);
    // rows that do not start on 16 bytes but on 8 (50 columns, say) go two floats at a time
    const bool padded = (flags & kPlanPadded) != 0;  // B is a copy with whole vectors, C stays as it is
    const bool pairs = !vec && !padded && (flags & kPlanNoPairs) == 0 && a->nnz <= kWholeRowEntries && pair_layout_ok(a);
    plan->VW = vec || padded ? 4 : (pairs ? 2 : 1);
    plan->ncolv = (a->Nd + plan->VW - 1) / plan->VW;
    const bool c_pairs = a->Nd % 2 == 0 && a->ldc % 2 == 0 && (reinterpret_cast<uintptr_t>(a->C) & 7u) == 0;
    plan->c_ragged = padded ? (c_pairs ? 2 : 1) : 0;
    plan->num_items = (long long)a->M + a->nnz;

    int kernel = a->kernel;
    bool forced = kernel != CSRSPMM_B200_KERNEL_AUTO;
    if (!forced) {
        kernel = forced_kernel_from_env();
        // an environment override that cannot run this layout falls back to AUTO
        if (kernel == CSRSPMM_B200_KERNEL_TMA && !tma_can_run(a)) kernel = CSRSPMM_B200_KERNEL_AUTO;
    }
    if (kernel == CSRSPMM_B200_KERNEL_AUTO) {
        // Measured on B200.  The bulk-copy path completes about one row copy per 80 cycles per SM, so it
        // only keeps HBM busy when a row of B is 2 KB (384 < Nd <= 512), where it is 3-4 % ahead of the merge
        // kernel -- provided B is far larger than L2, since an L2-resident B is served faster through the
        // load/store units.  Whole-row mapping wins when the longest row is known and close to the mean and B
        // comes from L2.  Beyond about 48 MB of B the time is the wait for HBM, and a lane group that stops at every
        // row end (bounds, columns, rows of B, store, each a round trip) asks for too little of it at once: the
        // merge kernel walks on across row ends (1 M rows of 16, 64 columns: 600 us against 812; 262 144 rows of 8:
        // 73 against 94; of 4: 51 against 74), unless rows are long enough to keep it busy by themselves (64 entries
        // of 128 columns: 773 against 745; 32 of 256: 1012 either way; 143 of 56: 703 against 601).  Everything else (unknown or skewed row lengths) takes
        // the merge kernel.  The entry point asked for does not change the choice.
        const double avg = a->M > 0 ? (double)a->nnz / (double)a->M : 0.0;
        const double b_bytes = (double)a->Kd * (double)a->Nd * 4.0;
        const bool rows_even = rows_known_even(a, avg);
        plan->rows_even = rows_even;
        if (tma_can_run(a) && a->Nd > 384 && b_bytes >= 1073741824.0 && !rows_even)
            kernel = CSRSPMM_B200_KERNEL_TMA;
        else if (rows_even && !rows_are_chains(a->M, avg, *plan) && (b_bytes < 48e6 || avg > 64.0 || (avg * a->Nd >= 8192.0 && a->Nd > 64)))
            kernel = CSRSPMM_B200_KERNEL_ROW;
        else
            kernel = CSRSPMM_B200_KERNEL_MERGE;
    }
    if (kernel == CSRSPMM_B200_KERNEL_TMA && !tma_can_run(a)) {
        set_last_error("the TMA kernel needs Nd %% 4 == 0, Nd <= 512, ldb/ldc %% 4 == 0 and "
                       "16-byte aligned B and C (Nd=%d ldb=%lld ldc=%lld)",
                       a->Nd, (long long)a->ldb, (long long)a->ldc);
        return CSRSPMM_B200_ERR_UNSUPPORTED;
    }
    plan->kernel = kernel;

    if (kernel == CSRSPMM_B200_KERNEL_TMA) {
        plan->G = 32;
        plan->NV = plan->ncolv <= 32 ? 1 : (plan->ncolv <= 64 ? 2 : 4);
        plan->shape = plan->NV == 1 ? 2 : (plan->NV == 2 ? 3 : 4);
        fill_split_geometry(a, plan, CSRSPMM_TUNE_MERGE_THREADS / 32, CSRSPMM_TUNE_TMA_TG);
        const size_t slot = align_up((size_t)a->Nd * 4, 128);
        size_t ring = (size_t)CSRSPMM_TUNE_TMA_SLOTS * slot;          // per warp
        if (ring < (size_t)512 * plan->NV) ring = (size_t)512 * plan->NV;  // must also hold the partial sums
        plan->tma_slot_bytes = slot;
        plan->dynamic_smem = (CSRSPMM_TUNE_MERGE_THREADS / 32) /*warps*/ * ring;
    } else {
        plan->shape = shape_for(plan->ncolv);
        plan->G = kShapes[plan->shape].G;
        plan->NV = kShapes[plan->shape].NV;
        plan->full = plan->VW == 4 && !padded && plan->G * plan->NV == plan->ncolv;
        if (CSRSPMM_TUNE_MERGE_NARROW && kernel == CSRSPMM_B200_KERNEL_MERGE && (flags & kPlanNoNarrow) == 0 && plan->ncolv >= 1 && plan->ncolv <= 4) {
            // one, two or four column vectors: lane groups of that many lanes (kNarrowShapes)
            plan->narrow = plan->ncolv == 1 ? 1 : (plan->ncolv == 2 ? 2 : 3);
            const ShapeDesc& ns = kNarrowShapes[plan->narrow - 1];
            plan->G = ns.G;
            plan->NV = ns.NV;
            plan->full = plan->VW == 4 && !padded && plan->G * plan->NV == plan->ncolv;
            const int groups = CSRSPMM_TUNE_MERGE_THREADS / ns.G;
            fill_split_geometry(a, plan, groups, merge_items_per_group(plan->num_items, groups, merge_min_blocks(1), ns.TG, coarse ? ns.TG : ns.G));
            plan->row_aligned = rows_fit_tiles(a, *plan, groups, ns.TG);
        } else if (kernel == CSRSPMM_B200_KERNEL_MERGE) {
            const int groups = CSRSPMM_TUNE_MERGE_THREADS / plan->G, most = kShapes[plan->shape].TG;
            const int least = coarse ? CSRSPMM_TUNE_MERGE_TG_SMALL : CSRSPMM_TUNE_MERGE_TG_LEAST;
            const int tg = merge_items_per_group(plan->num_items, groups, merge_min_blocks(plan->NV), most, least);
            plan->small_tile = tg <= CSRSPMM_TUNE_MERGE_TG_SMALL;
            fill_split_geometry(a, plan, groups, tg);
            plan->row_aligned = rows_fit_tiles(a, *plan, groups, most);
            if (plan->row_aligned && plan->small_tile) plan->small_tile = plan->tile + a->max_row_nnz + 1 <= groups * CSRSPMM_TUNE_MERGE_TG_SMALL;
        } else {
            const int groups = CSRSPMM_TUNE_ROW_THREADS / plan->G;
            plan->grid = ((long long)a->M + groups - 1) / groups;
            plan->any_count = a->nnz > kWholeRowEntries;
            plan->resident = (flags & kPlanNoPairs) == 0 && !padded && !plan->any_count ? resident_lanes(a, *plan) : 0;
            plan->short_rows = a->nnz <= (long long)CSRSPMM_TUNE_ROW_SHORT_MEAN * (long long)a->M;
            plan->low_occupancy = (long long)a->M * plan->G / 32 < (long long)kSms * 8;
#if CSRSPMM_TUNE_ROW_PERSISTENT > 0
            // many short rows: a CTA that lives for four 16-entry rows costs more to start than to
            // run (cfg2: 20.5 -> 18.6 us; 65536 rows of 13: 53 -> 45 us; long rows prefer the
            // finer dynamic balance of one CTA per few rows)
            if (a->nnz <= (long long)CSRSPMM_TUNE_ROW_PERSISTENT_MAX_MEAN * (long long)a->M && plan->grid > (long long)kSms * CSRSPMM_TUNE_ROW_PERSISTENT)
                plan->grid = (long long)kSms * CSRSPMM_TUNE_ROW_PERSISTENT;
#endif
            if (plan->VW == 4 && !plan->low_occupancy && !plan->short_rows) plan->row_build = row_build_for(plan->G, plan->NV, plan->full, plan->grid);
        }
    }
    // A next grid placed early goes where slots are free.  Behind a grid that fills the chip those are the slots
    // its CTAs leave, one by one and evenly; behind a smaller one they crowd on the SMs that had room, and the
    // crowded SMs finish late (4096 rows of 410 entries, 128 columns: 46.2 us per product against 43.4).
    const int resident_ctas = kernel == CSRSPMM_B200_KERNEL_ROW     ? (plan->low_occupancy ? 2 : plan->row_build ? row_build(plan->NV, plan->row_build).MINB : row_min_blocks(plan->NV))
                              : kernel == CSRSPMM_B200_KERNEL_MERGE ? merge_min_blocks(plan->NV)
                                                                    : CSRSPMM_TUNE_TMA_MINB;
    plan->fills_chip = plan->grid >= (long long)kSms * resident_ctas;
    if (plan->grid > 0x7fffffffLL) {
        set_last_error("grid of %lld CTAs exceeds the launch limit", plan->grid);
        return CSRSPMM_B200_ERR_UNSUPPORTED;
    }
    return CSRSPMM_B200_OK;
}

// The rules' figures are beside padded_b_bytes's declaration.
static bool odd_copy_pays(int Nd, double mean, double uses, double gather)
{
    return uses >= (Nd <= 256 ? 8.0 : 24.0) && gather >= 64e6 && (Nd >= 32 || mean <= 64.0);
}

static bool even_copy_pays(int M, int Nd, double mean, double uses, double gather, bool rows_even)
{
    if (gather < 250e6) return false;
    if (Nd <= 32) {
        constexpr int wave = kSms * CSRSPMM_TUNE_ROW_MINB_NV1 * (CSRSPMM_TUNE_ROW_THREADS / CSRSPMM_TUNE_S0_G);  // rows of eight lanes each
        return uses >= (Nd == 30 ? 16.0 : 48.0) && (mean <= 64.0 || M <= wave || M > wave + wave / 2);
    }
    const int pairs = Nd / 2, slots = pairs <= 32 ? 32 : (pairs <= 64 ? 64 : 128);
    const bool lanes_idle = Nd <= 256 && pairs * 100 <= slots * 85;
    return lanes_idle ? uses >= (slots == 128 || (slots == 32 && rows_even) ? 11.0 : 24.0) : uses >= 64.0 && Nd >= 96;
}

size_t padded_b_bytes(const csrspmm_b200_args* a)
{
    if (a->Nd % 4 == 0 || a->Nd < 17 || a->M <= 0 || a->Kd <= 0 || a->kernel == CSRSPMM_B200_KERNEL_TMA || a->nnz > kWholeRowEntries) return 0;
    const double mean = (double)a->nnz / a->M, uses = (double)a->nnz / a->Kd;
    const double gather = (double)a->nnz * a->Nd * 4.0;
    const bool pays = a->Nd % 2 ? odd_copy_pays(a->Nd, mean, uses, gather) : even_copy_pays(a->M, a->Nd, mean, uses, gather, rows_known_even(a, mean));
    return pays ? align_up((size_t)a->Kd * (size_t)((a->Nd + 3) / 4) * 16, 256) : 0;
}

int product_plan(const csrspmm_b200_args* a, Plan* plan)
{
    if (a != nullptr && a->struct_size == sizeof(csrspmm_b200_args) && a->workspace != nullptr &&
        (reinterpret_cast<uintptr_t>(a->workspace) & 255u) == 0) {
        const size_t pad = padded_b_bytes(a);
        if (pad > 0 && make_plan(a, plan, kPlanPadded) == CSRSPMM_B200_OK && padded_b_offset(*plan) + pad <= a->workspace_bytes)
            return CSRSPMM_B200_OK;
    }
    return make_plan(a, plan);
}

size_t worst_case_workspace(const csrspmm_b200_args* a)
{
    if (check_args(a, false) != CSRSPMM_B200_OK) return 0;
    // Most CTAs any split kernel takes: the bulk-copy kernel's fixed tile, or the merge kernel's waves of equal
    // tiles -- no more than the largest tile gives plus one wave, whatever the size, so the same bound holds for
    // every row block of the matrix.
    const long long items = (long long)a->M + a->nnz;
    Plan p;
    fill_split_geometry(a, &p, CSRSPMM_TUNE_MERGE_THREADS / 32, CSRSPMM_TUNE_TMA_TG);
    long long tiles = p.num_tiles;
    auto consider = [&](int groups, int most, int ctas_per_sm) {
        const long long t = items / ((long long)groups * most) + 1 + (long long)kSms * ctas_per_sm;
        if (t > tiles) tiles = t;
    };
    for (const ShapeDesc& k : kShapes) consider(CSRSPMM_TUNE_MERGE_THREADS / k.G, k.TG, merge_min_blocks(k.NV));
    for (const ShapeDesc& k : kNarrowShapes) consider(CSRSPMM_TUNE_MERGE_THREADS / k.G, k.TG, merge_min_blocks(1));
    if (items < tiles) tiles = items;  // no CTA without an item
    return align_up((size_t)tiles * sizeof(int32_t), 256) + (size_t)tiles * (size_t)p.carry_ld * sizeof(float);
}

}  // namespace csrspmm_b200
