// f64 state held in f32 / f32 state arithmetic / f32 fluxes
#include "od_launch_impl.cuh"

namespace od {
cudaError_t launch_stage_u64c32_narrow(const StageLaunch& L, cudaStream_t s) {
    return launch_stage_t<float, float, float, true>(L, s);
}
cudaError_t prepare_kernels_u64c32_narrow() { return prepare_t<float, float, float, true>(); }
}  // namespace od
