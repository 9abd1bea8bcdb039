// fp32_mixed.cu -- the batched FP32 forward over the tasks of mixed haplotypes (kBucketMixed, ghmm_internal.h).
namespace {
constexpr bool kMixedTasks = true;
}
#include "fp32_bucket.cuh"

namespace ghmm {

int launch_fp32_mixed(const DevTables &t, const DevBatch &b, int key, int grid, int block, cudaStream_t s) {
    return launch_fp32_form(t, b, key, grid, block, s);
}

int fp32_mixed_occupancy(int key, int block, int *blocks_per_sm) { return fp32_form_occupancy(key, block, blocks_per_sm); }

}  // namespace ghmm
