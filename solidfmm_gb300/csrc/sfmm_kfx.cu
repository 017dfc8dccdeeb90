// FP64 translations in 60-bit block fixed point (sfmm_fx.cuh).
#include "sfmm_kernel_impl.cuh"

namespace sfmm {
#define SHAPES(X, K) X(K, 4, 4) X(K, 4, 6) X(K, 4, 8) X(K, 8, 2) X(K, 8, 4) X(K, 8, 6) X(K, 8, 8)
#define KERNEL(G, ACC, HBM, WORK) (k_translate_fx<double, G, ACC, HBM, WORK>)
SFMM_DEFINE_LAUNCH(launch_translate_fx, occupancy_fx64, SHAPES, KERNEL)
}  // namespace sfmm
