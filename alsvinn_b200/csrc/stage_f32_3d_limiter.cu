// Stage-kernel instantiations for float precision, 3-D Euler, MC, MM and WENOF2.
#include "stage_dispatch.cuh"

namespace als {
cudaError_t launch_stage_f32_3d_limiter(ALS_STAGE_ARGS) {
    return launch_stage_group<float, 3, 2>(recon, flux, kind, shape, P, blocks_per_sm, s);
}
} // namespace als
