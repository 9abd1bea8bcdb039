// warp_list.cuh -- how a grid of warps takes the entries of a work list (pd.cu).  Internal linkage: each
// translation unit that includes it gets its own copy.
#pragma once
#include <cuda_runtime.h>

namespace ghmm {
namespace {

// Next entry of a work list for this warp: the first from the warp's place in the grid, warp w of every block before
// warp w + 1 of any, the following ones from an atomic cursor.  A list shorter than the grid then spreads over all SM
// sub-partitions; drawn by the cursor alone it goes to whichever blocks start first, up to three warps on one
// sub-partition while others stand idle, which for FP64 work (one FP64 pipe a sub-partition) costs as many times
// (the FP64 PD-HMM kernel on 100 pairs of 250 x 300 bases: 3.57 ms, spread 1.72; on 600 3.65 and 1.89; on 10,000, more
// than the grid has warps, 20.4 both ways).
__device__ __forceinline__ int draw_entry(int *cursor, bool &first, int lane) {
    if (first) {
        first = false;
        return (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
    }
    int t = 0;
    if (lane == 0) t = (int)(gridDim.x * (blockDim.x >> 5)) + atomicAdd(cursor, 1);
    return __shfl_sync(0xffffffffu, t, 0);
}

}  // namespace
}  // namespace ghmm
