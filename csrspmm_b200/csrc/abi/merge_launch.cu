// Starts the merge-path kernels (declared in launch.h).  One place for every entry point that runs
// them: csrspmm_b200_spmm, csrspmm_b200_spmm_noalloc, the row blocks and column panels of
// csrspmm_b200_spmm_host.  Stands where the reference's launchers fix their geometry
// (src/host/spmm_launcher.cu:63-70).
//
#include <cuda_runtime.h>

#include "../kernels/merge_kernel.cuh"
#include "launch.h"
#include "pdl.h"

namespace csrspmm_b200 {

namespace {

// A build with a column guard, with stores for a padded B's rows of C where that is what runs.
template <int G, int NV, int VW, int TG, int U, int FMT, bool PAIRS = VW == 4>
cudaError_t launch_guarded(const SpmmParams& p, const Plan& plan, cudaStream_t st)
{
    if constexpr (PAIRS)
        if (plan.c_ragged == kRaggedPairs)
            return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, U, FMT, false, false, kRaggedPairs>, (unsigned)plan.grid, kMergeThreads, 0, st, p);
    if (VW == 4 && plan.c_ragged == kRaggedFloats)
        return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, U, FMT, false, false, VW == 4 ? kRaggedFloats : 0>, (unsigned)plan.grid, kMergeThreads, 0, st, p);
    return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, U, FMT, false>, (unsigned)plan.grid, kMergeThreads, 0, st, p);
}

template <int S, int VW, int FMT>
cudaError_t launch_merge(const SpmmParams& p, const Plan& plan, cudaStream_t st)
{
    constexpr int G = kShapes[S].G, NV = kShapes[S].NV, TG = kShapes[S].TG;
    constexpr int TGS = CSRSPMM_TUNE_MERGE_TG_SMALL < TG ? CSRSPMM_TUNE_MERGE_TG_SMALL : TG;
    constexpr int U = merge_unroll(VW, NV);
    // one more row in flight where the grid is many waves long, hence waiting for HBM.  Six against five, 128 columns: 262 144
    // rows of 16 221.8 and 225.7 us, Zipf rows 221.2 and 229.5 (packed values 232.2 and 240.1), 200 000 Zipf rows 160.7 and
    // 165.2; 100 columns, 500 000 Zipf rows of 20 571 and 591; 64 columns, 1 M Zipf rows 605 and 610, 300 000 even ones 126.1
    // both; 48 columns 314.9 and 312.4.  Shorter grids the other way round: 47.5 and 45.2.
    constexpr int ULONG = VW == 4 && NV == 1 && G >= 16 ? CSRSPMM_TUNE_MERGE_U_LONG : U;
    const unsigned grid = (unsigned)plan.grid;
    if (ULONG != U && plan.tg == TG) {
        if (VW == 4 && plan.full) return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, ULONG, FMT, (VW == 4)>, grid, kMergeThreads, 0, st, p);
        return launch_guarded<G, NV, VW, TG, ULONG, FMT>(p, plan, st);
    }
    // Few items: smaller tiles, more CTAs.  A copy of B of even width is made for so many entries (padded_b_bytes) that only the
    // first and the last shape can have small tiles on one.
    constexpr bool kSmallPairs = VW == 4 && (S == 0 || S == 4);
    if (plan.small_tile && (kSmallPairs || plan.c_ragged != kRaggedPairs)) {
        if (VW == 4 && plan.full) return launch_overlapped(spmm_merge_kernel<G, NV, VW, TGS, U, FMT, (VW == 4)>, grid, kMergeThreads, 0, st, p);
        return launch_guarded<G, NV, VW, TGS, U, FMT, kSmallPairs>(p, plan, st);
    }
    if (VW == 4 && plan.full) return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, U, FMT, (VW == 4)>, grid, kMergeThreads, 0, st, p);
    return launch_guarded<G, NV, VW, TG, U, FMT>(p, plan, st);
}

// Very narrow dense operands: lane groups of 1, 2 or 4 lanes (kNarrowShapes).  No padded copy is this narrow, and with 16-byte
// vectors one or two lanes have a column each; only three vectors leave a lane idle.
template <int K, int VW, int FMT>
cudaError_t launch_merge_narrow(const SpmmParams& p, const Plan& plan, cudaStream_t st)
{
    constexpr int G = kNarrowShapes[K].G, NV = kNarrowShapes[K].NV, TG = kNarrowShapes[K].TG;
    constexpr int U = merge_unroll(VW, NV);
    const unsigned grid = (unsigned)plan.grid;
    if (VW == 4 && (G < 4 || plan.full)) return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, U, FMT, (VW == 4)>, grid, kMergeThreads, 0, st, p);
    if constexpr (VW != 4 || G == 4) return launch_overlapped(spmm_merge_kernel<G, NV, VW, TG, U, FMT, false>, grid, kMergeThreads, 0, st, p);
    return cudaErrorInvalidValue;
}

template <int VW, int FMT>
cudaError_t dispatch_merge(const SpmmParams& p, const Plan& plan, cudaStream_t st)
{
    switch (plan.narrow) {
        case 1: return launch_merge_narrow<0, VW, FMT>(p, plan, st);
        case 2: return launch_merge_narrow<1, VW, FMT>(p, plan, st);
        case 3: return launch_merge_narrow<2, VW, FMT>(p, plan, st);
        default: break;
    }
    switch (plan.shape) {
        case 0: return launch_merge<0, VW, FMT>(p, plan, st);
        case 1: return launch_merge<1, VW, FMT>(p, plan, st);
        case 2: return launch_merge<2, VW, FMT>(p, plan, st);
        case 3: return launch_merge<3, VW, FMT>(p, plan, st);
        default: return launch_merge<4, VW, FMT>(p, plan, st);
    }
}

}  // namespace

cudaError_t launch_merge_kernel(const SpmmParams& p, const Plan& plan, bool e2m1, cudaStream_t st)
{
    if (plan.VW == 4) return e2m1 ? dispatch_merge<4, kValuesE2M1>(p, plan, st) : dispatch_merge<4, kValuesF32>(p, plan, st);
    if (plan.VW == 2) return e2m1 ? dispatch_merge<2, kValuesE2M1>(p, plan, st) : dispatch_merge<2, kValuesF32>(p, plan, st);
    return e2m1 ? dispatch_merge<1, kValuesE2M1>(p, plan, st) : dispatch_merge<1, kValuesF32>(p, plan, st);
}

cudaError_t launch_fixup_kernel(const SpmmParams& p, const Plan& plan, cudaStream_t st)
{
    const int warps = 256 / 32;
    const unsigned grid = (unsigned)((plan.num_tiles + warps - 1) / warps);
    if (plan.c_ragged) {  // carries lie column by column, and C is not aligned to their vectors: added float by float (also pairs)
        SpmmParams q = p;
        q.ncolv = p.Nd;
        return launch_overlapped(spmm_fixup_kernel<1>, grid, 256, 0, st, q, (int)plan.num_tiles);
    }
    return launch_overlapped(plan.VW == 4 ? spmm_fixup_kernel<4> : plan.VW == 2 ? spmm_fixup_kernel<2> : spmm_fixup_kernel<1>, grid, 256, 0, st, p, (int)plan.num_tiles);
}

}  // namespace csrspmm_b200
