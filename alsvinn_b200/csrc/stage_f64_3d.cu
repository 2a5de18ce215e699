// Stage-kernel instantiations for double precision, 3-D Euler.
#include "stage_dispatch.cuh"

namespace als {
cudaError_t launch_stage_f64_3d(ALS_STAGE_ARGS) {
    static const StageLauncher units[kReconGroups] = {launch_stage_group<double, 3, 0>,
        launch_stage_f64_3d_eno, launch_stage_f64_3d_limiter};
    return launch_stage_unit(units, recon, flux, kind, shape, P, blocks_per_sm, s);
}

void stage_tile_f64_3d(int shape, int* tile) {
    stage_tile_dim<3>(shape, tile);
}
} // namespace als
