// Table layout of the 60-bit fixed-point kernel that the host builder and the
// kernel share (no CUDA headers: the builder is tested without them).
#pragma once

#ifdef __CUDACC__
#define SFMM_HD __host__ __device__
#else
#define SFMM_HD
#endif

namespace sfmm {

// doubles per row (input degree) of a z matrix with L outputs, for G threads
// per translation: pairs of G/2-row blocks
SFMM_HD constexpr int fx_hrow(int L, int G) { return ((L + G / 2 - 1) / (G / 2) + 1) / 2 * G; }

}  // namespace sfmm
