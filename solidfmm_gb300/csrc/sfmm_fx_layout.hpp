// Table layout of the 60-bit fixed-point kernel that the host builder and the
// kernel share (no CUDA headers: the builder is tested without them).
#pragma once

#ifdef __CUDACC__
#define SFMM_HD __host__ __device__
#else
#define SFMM_HD
#endif

namespace sfmm {

// elements per row (input degree) of a z matrix with L outputs, for G threads
// per translation: vectors of V blocks of G/2 rows
SFMM_HD constexpr int fx_hrow(int L, int G, int V = 2) { return ((L + G / 2 - 1) / (G / 2) + V - 1) / V * (G / 2) * V; }

}  // namespace sfmm
