// Fused translation kernels, float arithmetic (sfmm_f32.cuh).
#include "sfmm_kernel_impl.cuh"

namespace sfmm {
cudaError_t launch_translate_32(const KParams &p, const LaunchShape &s, int grid, cudaStream_t st)
{
    return launch_fx<float>(p, s, grid, st);
}
int occupancy_32(const LaunchShape &s) { return occupancy_fx<float>(s); }
}  // namespace sfmm
