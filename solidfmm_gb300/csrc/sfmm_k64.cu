// FP64 translations above order 32, one warp per translation.
#include "sfmm_kernel_impl.cuh"

namespace sfmm {
#define SHAPES(X, K) X(K, 32, 2) X(K, 32, 3)
#define KERNEL(G, ACC, HBM, WORK) (k_translate<double, G, ACC, false, HBM, WORK>)
SFMM_DEFINE_LAUNCH(launch_translate_64, occupancy_64, SHAPES, KERNEL)
}  // namespace sfmm
