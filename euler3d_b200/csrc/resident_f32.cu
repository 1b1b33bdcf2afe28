// Resident kernel, FP32_FLUX.
#include "common.hpp"
#include "stage_resident.cuh"

namespace e3d {

int resident_max_blocks_f32(int shape, size_t smem) { return ResidentLaunch<PREC_F32>::max_blocks(shape, smem); }

bool launch_resident_f32(const StageArgs &a, const ResidentArgs &r, int shape, size_t smem, cudaStream_t s) {
    return ResidentLaunch<PREC_F32>::launch(a, r, shape, smem, s);
}

}  // namespace e3d
