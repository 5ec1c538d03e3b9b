// Which staged row a thread of the ensemble's force loop reads, as index arithmetic without a device.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

namespace gtd {

// Threads that take `rows` rows, ib each: the smallest multiple of 32 with ib * threads >= rows.
__host__ __device__ __forceinline__ int ens_row_threads(int rows, int ib) { return ((rows + ib - 1) / ib + 31) & ~31; }

// The row a thread stands on for its i-th candidate i: a thread without a row there repeats its first, r0,
// whose fold of bodies its warp goes through anyway, and where r0 is past the rows [.., nc) as well (fewer
// than 32 rows) the last row.  Results of rows at or past nc are dropped.
__host__ __device__ __forceinline__ int ens_stand_in(int i, int r0, int nc) { return i < nc ? i : r0; }
__host__ __device__ __forceinline__ int ens_staged_row(int i, int r0, int nc) {
    const int k = ens_stand_in(i, r0, nc);
    return k < nc ? k : nc - 1;
}

// Floats of a staged coordinate array: the largest system, even.
inline int ens_stride(int max_n) { return std::max(2, (max_n + 1) & ~1); }

}  // namespace gtd
