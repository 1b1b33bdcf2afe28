// Resident kernel, FP64_EXACT.
#include "common.hpp"
#include "stage_resident.cuh"

namespace e3d {

int resident_max_blocks_exact(int shape, size_t smem) { return ResidentLaunch<PREC_EXACT>::max_blocks(shape, smem); }

bool launch_resident_exact(const StageArgs &a, const ResidentArgs &r, int shape, size_t smem, cudaStream_t s) {
    return ResidentLaunch<PREC_EXACT>::launch(a, r, shape, smem, s);
}

}  // namespace e3d
