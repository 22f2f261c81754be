// Resident kernel: a column panel of B in shared memory, every row of A against it.
//
// Serves the reference's whole-row kernels (src/device/csrspmm_warp_per_row_smem_fp4.cu:11-84 and its siblings) where A
// has few columns and B is wide: the layer shapes of its torch benchmark (torch_csrspmm/torch_benchmarks.py:15-20:
// 64 to 256 columns of A, 1024 to 4096 of B).  There each row of B is named by many rows of A, and gathering it from
// L2 every time is what the row kernel's time is: 3.4 GB for a 16 MB result (8192 x 256 at 10 %, 4096 columns), 15 to 17
// TB/s.  A CTA here keeps Kd x TC floats of B in shared memory, and the gather is one 128-byte wavefront per eight lanes.
//
// TC = 4 * G columns: a lane group of G lanes owns one row at a time and a float4 of its columns.  G = 32 takes A of
// up to 400 columns, G = 16 up to 800; narrower panels would spend the gain on (column, value) reads and on groups of a
// warp that wait for each other.  One CTA of 1024 threads per SM.  The (panel, row) pairs, panel by panel, are cut into
// as many equal runs as there are CTAs, so that every SM has the same share whatever the numbers of panels and rows.
//
// (column, value) come a chunk of 32 at a time: the next chunk -- of the same row or of the group's next one -- is
// requested before the current one is used, its columns turned into byte offsets and both put in shared memory, from
// where two entries are read at a time.  What bounds it: shared-memory wavefronts, 4 for the row of B and half of one for
// the entry per 128 products.  8192 x 256 at 10 % times 4096 columns: 4.85 wavefronts are counted and 5.8 cycles taken; the
// pipe is 89.5 % busy, 83.6 % with shared memory and 6 % with A and C.
// Against the row kernel there: 10 % dense 198 -> 140 us, 30 % 460 -> 379, 5 % 112 -> 87; 1024 x 128 times 2048 columns at
// 10 % 16.4 -> 9.8; 16 000 x 700 times 600, rows of 100 (G = 16) 260 -> 204.
//
// Each output is one sequential sum over the row's entries in stored order, as in the row kernel.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "tuning.h"

namespace csrspmm_b200 {

namespace cg = cooperative_groups;

constexpr int kResidentThreads = 1024;
constexpr int kResidentChunk = 32;
constexpr int kResidentSlice = kResidentChunk + 2;  // int2 per group: groups of a warp read different banks
constexpr int kResidentPanelBytes = 200 * 1024;  // of B, at most

template <int G>
constexpr int resident_smem_bytes(int Kd)
{
    return Kd * (G * 16) + (kResidentThreads / G) * kResidentSlice * (int)sizeof(int2);
}

// total = panels * M; CTA b takes pairs [b * total / grid, (b + 1) * total / grid).
template <int G, int FMT>
__global__ void __launch_bounds__(kResidentThreads, 1) spmm_resident_kernel(const SpmmParams p, const long long total)
{
    wait_for_previous_grid();
    if (p.release_early) release_next_grid();
    constexpr int GROUPS = kResidentThreads / G;
    constexpr int CHUNK = kResidentChunk;
    constexpr int PAIRS = CHUNK / G;  // (col, val) pairs a lane fetches per chunk
    extern __shared__ __align__(128) unsigned char smem[];
    int2* const all_cv = reinterpret_cast<int2*>(smem);
    float4* const panel = reinterpret_cast<float4*>(all_cv + GROUPS * kResidentSlice);

    const cg::thread_block_tile<G> tile = cg::tiled_partition<G>(cg::this_thread_block());
    const int lane = tile.thread_rank();
    const int g = threadIdx.x / G;
    int2* const cv = all_cv + g * kResidentSlice;
    const unsigned char* const b_lane = reinterpret_cast<const unsigned char*>(panel + lane);

    const long long u0 = total * blockIdx.x / gridDim.x, u1 = total * (blockIdx.x + 1) / gridDim.x;
    for (long long u = u0; u < u1;) {
        const int t = (int)(u / p.M);
        const int row0 = (int)(u - (long long)t * p.M);
        const int row1 = (int)min((long long)p.M, row0 + (u1 - u));
        u += row1 - row0;

        // ---- the panel -------------------------------------------------------------------------
        __syncthreads();  // the last panel is done with
        const int cv0 = t * G;  // its first column vector
        for (int k = threadIdx.x; k < p.Kd * G; k += kResidentThreads) {
            const int r = k / G, c = cv0 + k % G;
            if (c < p.ncolv) async_copy_vec<4>(smem_addr(panel + k), p.B + (long long)r * p.ldb + 4LL * c);
        }
        async_commit();

        // ---- the group's rows: row0 + g, + GROUPS, ... ------------------------------------------
        int row = row0 + g;
        // clamped so that a malformed row_ptr stays inside the arrays; at most kWholeRowEntries, as in the row kernel
        auto bounds = [&](int r, int& first, int& last) {
            first = last = 0;
            if (r < row1) {
                first = max(__ldg(p.row_ptr + r) - p.rp_base, 0);
                last = min(__ldg(p.row_ptr + r + 1) - p.rp_base, p.nnz);
            }
        };
        int c_next[PAIRS];
        float a_next[PAIRS];
        auto request = [&](int base, int last) {
#pragma unroll
            for (int q = 0; q < PAIRS; ++q) {
                const int j = base + q * G + lane;
                c_next[q] = 0;
                a_next[q] = 0.f;
                if (j < last) {
                    int c = __ldcs(p.col_idx + j);
                    a_next[q] = load_value<FMT>(p.values, j, p.value_scale);
                    if ((unsigned)c >= (unsigned)p.Kd) {  // never fault on a bad index
                        c = min(max(c, 0), p.Kd - 1);
                        report_status(p, kStatusColClamped);
                    }
                    c_next[q] = c;
                }
            }
        };
        int j, last, next_first, next_last;
        bounds(row, j, last);
        bounds(row + GROUPS, next_first, next_last);
        request(j, last);
        async_wait<0>();
        __syncthreads();

        Vec<4> acc[1];
        acc[0].zero();
        while (row < row1) {
            tile.sync();  // the previous chunk has been consumed by every lane of the group
#pragma unroll
            for (int q = 0; q < PAIRS; ++q) cv[q * G + lane] = make_int2(c_next[q] * (G * 16), __float_as_int(a_next[q]));
            tile.sync();
            const int n = min(CHUNK, last - j);
            const bool ends = j + CHUNK >= last;
            if (ends) request(next_first, next_last);
            else request(j + CHUNK, last);
            auto step = [&](int off, int bits) {
                Vec<4> b;
                b.v = *reinterpret_cast<const float4*>(b_lane + off);
                acc[0].fma(__int_as_float(bits), b);
            };
            int e = 0;
            for (; e + 4 <= n; e += 4) {
                const int4 x = *reinterpret_cast<const int4*>(cv + e), y = *reinterpret_cast<const int4*>(cv + e + 2);
                step(x.x, x.y);
                step(x.z, x.w);
                step(y.x, y.y);
                step(y.z, y.w);
            }
            for (; e < n; ++e) step(cv[e].x, cv[e].y);
            if (ends) {
                store_row<G, 1, 4>(p, row, cv0, lane, acc);
                acc[0].zero();
                row += GROUPS;
                j = next_first;
                last = next_last;
                bounds(row + GROUPS, next_first, next_last);
            } else {
                j += CHUNK;
            }
        }
    }
}

}  // namespace csrspmm_b200
