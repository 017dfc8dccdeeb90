// Split-precision translations (sfmm_split.cuh).
#include "sfmm_kernel_impl.cuh"

namespace sfmm {
#define SHAPES(X, K) X(K, 4, 1) X(K, 4, 2) X(K, 4, 4) X(K, 4, 6) X(K, 4, 8) X(K, 8, 1) X(K, 8, 2) X(K, 8, 3) X(K, 8, 4)
#define KERNEL(G, ACC, HBM, WORK) (k_translate_split<G, ACC, HBM, WORK>)
SFMM_DEFINE_LAUNCH(launch_translate_ffq, occupancy_ffq, SHAPES, KERNEL)
}  // namespace sfmm
