// FP32 translations (sfmm_f32.cuh).
#include "sfmm_kernel_impl.cuh"

namespace sfmm {
#define SHAPES(X, K) X(K, 4, 4) X(K, 4, 6) X(K, 4, 8) X(K, 4, 10) X(K, 4, 14) X(K, 8, 4) X(K, 8, 6) X(K, 8, 8)
#define KERNEL(G, ACC, HBM, WORK) (k_translate_fx<float, G, ACC, HBM, WORK>)
SFMM_DEFINE_LAUNCH(launch_translate_32, occupancy_32, SHAPES, KERNEL)
}  // namespace sfmm
