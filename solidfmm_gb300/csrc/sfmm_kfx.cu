// Fused translation kernels, FP64 in 60-bit block fixed point (sfmm_fx.cuh).
#include "sfmm_kernel_impl.cuh"

namespace sfmm {
cudaError_t launch_translate_fx(const KParams &p, const LaunchShape &s, int grid, cudaStream_t st)
{
    return launch_fx<double>(p, s, grid, st);
}
int occupancy_fx64(const LaunchShape &s) { return occupancy_fx<double>(s); }
}  // namespace sfmm
