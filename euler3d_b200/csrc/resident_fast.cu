// Resident kernel, FP64.
#include "common.hpp"
#include "stage_resident.cuh"

namespace e3d {

int resident_max_blocks_fast(int shape, size_t smem) { return ResidentLaunch<PREC_FAST>::max_blocks(shape, smem); }

bool launch_resident_fast(const StageArgs &a, const ResidentArgs &r, int shape, size_t smem, cudaStream_t s) {
    return ResidentLaunch<PREC_FAST>::launch(a, r, shape, smem, s);
}

}  // namespace e3d
