// Stage-kernel instantiations for float precision, 2-D Euler.
#include "stage_dispatch.cuh"

namespace als {
cudaError_t launch_stage_f32_2d(ALS_STAGE_ARGS) {
    static const StageLauncher units[kReconGroups] = {launch_stage_group<float, 2, 0>,
        launch_stage_f32_2d_eno, launch_stage_f32_2d_limiter};
    return launch_stage_unit(units, recon, flux, kind, shape, P, blocks_per_sm, s);
}

void stage_tile_f32_2d(int shape, int* tile) {
    stage_tile_dim<2>(shape, tile);
}
} // namespace als
