// Launch and occupancy of the fused translation kernels; included by
// sfmm_k64.cu (FP64 above order 32), sfmm_kfx.cu (FP64 up to 32), sfmm_k32.cu
// (FP32) and sfmm_kffq.cu (split), one translation unit each, compiled in
// parallel.  An instance is a group size G and a number ACC of row blocks per
// thread, the block count of the launch's order rounded up to an instantiated
// one, in three forms: expansions in device memory, in host memory read over
// the link, and tiles from a work list.
#pragma once

#include "sfmm_launch.hpp"
#include "sfmm_translate.cuh"

namespace sfmm {

// Launch shapes come from best_shape, whose occupancy query (below) has set
// the kernels' shared-memory limit on the current device, so a launch (also
// inside a CUDA graph capture) makes no other runtime call.
using Kernel = void (*)(KParams);

static cudaError_t launch_inst(Kernel hbm, Kernel host, Kernel work, const KParams &p, const LaunchShape &s, int grid,
                               cudaStream_t st)
{
    clear_stale_error();
    if (p.work && !p.in_hbm) return cudaErrorInvalidValue;  // work lists are a device-memory form
    const Kernel k = p.work ? work : p.in_hbm ? hbm : host;
    k<<<grid, s.threads, s.smem, st>>>(p);
    return cudaGetLastError();
}

// resident CTAs per SM of the device-memory instance (the shape's grid
// sizing); the host-memory and work-list instances are set up alongside
static int occupancy_inst(Kernel hbm, Kernel host, Kernel work, const LaunchShape &s)
{
    for (Kernel k : {hbm, host, work}) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, hbm, s.threads, s.smem) != cudaSuccess) return 0;
    return nb;
}

// Defines launch and occupancy functions over the instances of SHAPES, KERNEL(G, ACC, HBM, WORK) one of them.
#define SFMM_DEFINE_LAUNCH(LAUNCH, OCCUPANCY, SHAPES, KERNEL)                                               \
    cudaError_t LAUNCH(const KParams &p, const LaunchShape &s, int grid, cudaStream_t st)                    \
    {                                                                                                        \
        SHAPES(SFMM_LAUNCH_ONE, KERNEL)                                                                      \
        return cudaErrorInvalidValue;                                                                        \
    }                                                                                                        \
    int OCCUPANCY(const LaunchShape &s)                                                                      \
    {                                                                                                        \
        SHAPES(SFMM_OCCUPANCY_ONE, KERNEL)                                                                   \
        return 0;                                                                                            \
    }
#define SFMM_LAUNCH_ONE(KERNEL, G_, A_)                                                                      \
    if (s.G == G_ && s.acc == A_)                                                                            \
        return launch_inst(KERNEL(G_, A_, true, false), KERNEL(G_, A_, false, false), KERNEL(G_, A_, true, true), p, s, \
                           grid, st);
#define SFMM_OCCUPANCY_ONE(KERNEL, G_, A_)                                                                   \
    if (s.G == G_ && s.acc == A_)                                                                            \
        return occupancy_inst(KERNEL(G_, A_, true, false), KERNEL(G_, A_, false, false), KERNEL(G_, A_, true, true), s);

}  // namespace sfmm
