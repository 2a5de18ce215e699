// Stage-kernel instantiations for float precision, 2-D Euler, the wide stencils (ENO3, ENO4, WENO3).
#include "stage_dispatch.cuh"

namespace als {
cudaError_t launch_stage_f32_2d_eno(ALS_STAGE_ARGS) {
    return launch_stage_group<float, 2, 1>(recon, flux, kind, shape, P, blocks_per_sm, s);
}
} // namespace als
