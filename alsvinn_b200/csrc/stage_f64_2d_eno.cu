// Stage-kernel instantiations for double precision, 2-D Euler, the wide stencils (ENO3, ENO4, WENO3).
#include "stage_dispatch.cuh"

namespace als {
cudaError_t launch_stage_f64_2d_eno(ALS_STAGE_ARGS) {
    return launch_stage_group<double, 2, 1>(recon, flux, kind, shape, P, blocks_per_sm, s);
}
} // namespace als
