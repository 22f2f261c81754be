// See scan.h.
#include "scan.h"

#include "../kernels/scan_kernels.cuh"
#include "pdl.h"

namespace csrspmm_b200 {

static long long scan_tiles(long long n) { return n > 0 ? (n + kScanTile - 1) / kScanTile : 1; }

size_t scan_scratch_bytes(long long n) { return (size_t)scan_tiles(n) * (sizeof(long long) + sizeof(int)); }

cudaError_t exclusive_scan(const int* counts, long long n, int* offsets, void* scratch, long long* results, cudaStream_t st)
{
    const long long tiles = scan_tiles(n);
    long long* tile_sum = static_cast<long long*>(scratch);
    int* tile_max = reinterpret_cast<int*>(tile_sum + tiles);
    cudaError_t e = launch_overlapped(scan_tiles_kernel, (unsigned)tiles, kScanThreads, 0, st, counts, n, offsets, tile_sum, tile_max, results);
    if (e == cudaSuccess && tiles > 1)
        e = launch_overlapped(scan_finish_kernel, (unsigned)tiles, kScanThreads, 0, st, n, offsets, tile_sum, tile_max, results);
    return e;
}

}  // namespace csrspmm_b200
