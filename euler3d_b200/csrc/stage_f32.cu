// FP32_FLUX instantiations of the face-tile stage kernel.
#include "common.hpp"
#include "stage_ws.cuh"

namespace e3d {

void prepare_tile_f32(size_t smem_bytes, size_t ws_smem_bytes) {
    raise_smem_limit((const void *)tile_kernel_f32<4>, with_forces(smem_bytes, 1));
    raise_smem_limit((const void *)tile_kernel_f32<9>, with_forces(smem_bytes, 1));
    raise_smem_limit((const void *)tile_kernel_f32<4, true>, with_forces(smem_bytes, 1));
    if (ws_smem_bytes) raise_smem_limit((const void *)tile_ws_kernel<WS_F32>, ws_smem_bytes);
}

void prepare_batch_f32(size_t smem_bytes, size_t ws_smem_bytes) {
    raise_smem_limit((const void *)tile_batch_kernel_f32<8>, smem_bytes);
    raise_smem_limit((const void *)tile_batch_kernel_f32<4, true>, smem_bytes);
    if (ws_smem_bytes) raise_smem_limit((const void *)tile_ws_batch_kernel<WS_F32>, ws_smem_bytes);
}

// One stage of every member of a batch with the warp-specialised persistent kernel.
void launch_batch_ws_f32(const BatchStage &bs, int grid, size_t smem_bytes, cudaStream_t s) {
    tile_ws_batch_kernel<WS_F32><<<grid, kWsThreads, smem_bytes, s>>>(bs);
}

// One stage of every member of a batch: `grid` blocks over the (member, tile) table.
void launch_batch_f32(const BatchStage &bs, bool many_faces, int grid, size_t smem_bytes, cudaStream_t s) {
    launch_dependent(many_faces ? tile_batch_kernel_f32<4, true> : tile_batch_kernel_f32<8>, grid, kStageThreads, smem_bytes,
                     s, bs);
}

// variant 2: face tiles with registers for four blocks/SM; 3: warp-specialised persistent face
// tiles; 4: face tiles at nine blocks/SM (56 registers, no spills; 1.57M tetrahedra 71.7 us a stage at
// eight blocks, 69.5 at nine, 561k-cell AUSM channel 25.0 and 23.4; the batch kernel spills at nine and
// takes 141 us an iteration instead of 131, so it stays at eight; an iteration's first stage runs at eight
// too where it carries force blocks, whose 24 KB are more than a tile's 17.8)
void launch_stage_f32(const StageArgs &a, const CoeffArgs &c, cudaStream_t s, int variant) {
    const int blocks = (a.n_cells + kStageThreads - 1) / kStageThreads;
    const size_t smem = tile32_smem_bytes(a.smem_cells, a.smem_faces, a.max_contrib);
    if (a.max_contrib > kElementFaces) {  // one kernel for meshes with cells of more faces
        launch_dependent(tile_kernel_f32<4, true>, blocks + a.force_blocks, kStageThreads, with_forces(smem, a.force_blocks), s,
                         a, c);
    } else if (variant == 3) {
        const size_t ws = ws_smem_for(ws_buffer_bytes(WS_F32, a.smem_cells, a.smem_faces, a.max_contrib), a.ws_buffers);
        tile_ws_kernel<WS_F32><<<a.pipe_grid, kWsThreads, ws, s>>>(a);
    } else if (variant == 4) {
        launch_dependent(tile_kernel_f32<9>, blocks + a.force_blocks, kStageThreads, with_forces(smem, a.force_blocks), s, a, c);
    } else {
        launch_dependent(tile_kernel_f32<4>, blocks + a.force_blocks, kStageThreads, with_forces(smem, a.force_blocks), s, a, c);
    }
}

}  // namespace e3d
