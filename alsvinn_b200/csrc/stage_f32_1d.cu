// Stage-kernel instantiations for float precision, 1-D Euler.
#include "stage_dispatch.cuh"

namespace als {
cudaError_t launch_stage_f32_1d(ALS_STAGE_ARGS) {
    static const StageLauncher units[kReconGroups] = {launch_stage_group<float, 1, 0>,
        launch_stage_group<float, 1, 1>, launch_stage_group<float, 1, 2>};
    return launch_stage_unit(units, recon, flux, kind, shape, P, blocks_per_sm, s);
}

void stage_tile_f32_1d(int shape, int* tile) {
    stage_tile_dim<1>(shape, tile);
}

cudaError_t launch_line_f32(int recon, int flux, ALS_LINE_ARGS) {
    return launch_line<float>(recon, flux, rk3, P, members, blocks, s, clusters);
}
} // namespace als
