// Host-side operator tables for the GPU translation kernels.
//
// Plays the role of the reference's operator_data<real> (factorials and the
// packed real/imag swap matrices, solidfmm/operator_data.cpp:48-244), built
// once per context in FP64 and uploaded.  The kernels work in an orthogonal
// basis of each degree-n subspace:
//
//   D_m   = sqrt((n-m)! (n+m)!),   s_0 = sqrt(2), s_m = 1 (m > 0)
//   E_m   = D_m / s_m,             F_m = D_m * s_m
//   W_R   = E Rf E^-1 = F^-1 Rt F  (Rf, Rt: the reference's real swap matrix and its
//                                   transposed variant, operator_data.cpp:48-122)
//   W_I   = D If D^-1 = D^-1 It D  (imag swap matrix, operator_data.cpp:74-147)
//
// W_R and W_I are orthogonal, symmetric involutions with entries |w| <= 1, so
// both the forward (Rf) and backward (Rt) swaps use the same W.  The diagonal
// scalings are folded into the edge factors (first and last rotation of each
// degree) and into the z-translation matrices H_m.
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

namespace sfmm {

struct HostTables {
    int P = 0;
    // W for degree n (d = n+1) at woff[n].  Only the checkerboard a swap
    // uses is stored: W_R(i, j) is nonzero only for j = jr(i) + 2t with
    // jr(i) = (i+n) & 1, W_I(i, j) only for j = ji(i) + 2t with
    // ji(i) = jr(i) ^ 1.  Slot t holds R = wrows(d,pad) rows of W_R (row i at
    // 2tR + i) followed by R rows of W_I (at 2tR + R + i).  Rows are padded
    // to a multiple of row_pad(P) and slots to wcols(d) = (d+3)/2 with zeros
    // (the swap loops prefetch one slot past the last column), so the
    // kernels load coefficients without bounds checks.
    int pad = 8;
    std::vector<double> W;
    std::vector<int> woff;
    // The blocks of degrees below 32 padded to 8 rows, of orders above 32 (pad
    // 32) only.  No kernel reads them: launches at order bounds up to 32 take
    // FxTables and its like below.
    std::vector<double> W8;
    std::vector<int> woff8;
    // Edge factors indexed n(n+1)/2 + m:
    std::vector<double> e_in_M;   // E^(n)_m        forward of M2M/M2L inputs
    std::vector<double> e_in_L;   // 1 / F^(n)_m    forward of L2L inputs
    std::vector<double> e_out_L;  // F^(n)_m        backward of M2L/L2L outputs
    std::vector<double> e_out_M;  // 1 / E^(n)_m    backward of M2M outputs
    // z-translation matrices per op (0 M2M, 1 M2L, 2 L2L) and column m:
    // entry (output n', input k) at hoff[m] + (k-m)*hrows(P-m,pad) + (n'-m),
    // output rows padded with zeros to a multiple of row_pad(P).
    std::vector<double> H[3];
    std::vector<int> hoff;
};

// Dehnen's swap matrix B_n^{m,l} (swap_matrix.cpp:149-171), all n < P,
// stored per n as (2n+1)^2 with (m,l) at (m+n) + (l+n)(2n+1).
std::vector<std::vector<double>> swap_matrices(int P);

// Row padding of the coefficient blocks: 8 when the kernels run 4 threads
// per translation (orders up to 32), 32 when they run one warp per
// translation (larger orders).
inline int row_pad(int P) { return P <= 32 ? 8 : 32; }
inline int wrows(int d, int pad) { return (d + pad - 1) & ~(pad - 1); }
inline int wcols(int d) { return (d + 3) / 2; }
// W_R (part 0) or W_I (part 1) of degree n at (row i, column j), from the
// compact layout
double w_entry(const HostTables &t, int n, int part, int i, int j);
inline int hrows(int L, int pad) { return (L + pad - 1) & ~(pad - 1); }

HostTables build_tables(int P);

// Tables of the 60-bit fixed-point kernel for G threads per translation and
// orders up to P, from the context's tables.
struct FxTables {
    int P = 0;
    // Swap coefficients round(w 2^60) = h 2^30 + l, |l| <= 2^29, as (h, l)
    // pairs; degree n at woff[n] (in pairs).  Lane q of the G lanes holds part
    // q & 1 (W_R, W_I) of the rows i = (q >> 1) + (G/2) a, a < NA =
    // ceil(d / (G/2)); slot t (column ((i + n + part) & 1) + 2t) lies at
    // woff[n] + t NA G: for each pair of rows a = 2p, 2p + 1 the two
    // coefficients of lane q at (p G + q) 2, for an odd last row lane q's at
    // (NA - 1) G + q.  Slots t < (d + 1) / 2.
    std::vector<int32_t> W;
    std::vector<int> woff;
    // z matrices in FP64: column m of op at hoff[m], row k of it
    // (k - m) fx_hrow(P - m, G) further, output n' = m + r + (G/2) b at
    // (b / 2) G + 2 r + (b & 1)
    std::vector<double> H[3];
    std::vector<int> hoff;
};
FxTables build_fx_tables(const HostTables &t, int G, int P);
// The same tables for the FP32 kernel: swap coefficients in FP32, degree n at
// woff[n], slot t 4 NQ G further (NQ = ceil(NA / 4)), lane q's rows a at
// (a / 4) 4 G + 4 q + a % 4; z matrices in FP32, output n' at
// (b / 4) 2 G + 4 r + b % 4 of a row of fx_hrow(P - m, G, 4) elements.
struct F32Tables {
    std::vector<float> W, H[3];
    std::vector<int> woff, hoff;
};
F32Tables build_f32_tables(const HostTables &t, int G, int P);
// Tables of the split kernel: swap coefficients round(w 2^30) as (W_R, W_I)
// pairs, degree n at woff[n] (in pairs, one more slot after the last), slot t (column jr + 2t of W_R, (jr ^
// 1) + 2t of W_I, jr = (q + n) & 1) NA G further, rows i = q + G a of lane q:
// for each pair a = 2p, 2p + 1 at (p G + q) 2, an odd last row at (NA - 1) G + q.
// z matrices as float-float pairs (hi, lo), output n' = m + q + G b at (b / 2)
// 2 G + 2 q + (b & 1) of a row of fx_hrow(P - m, 2 G) entries.
struct SplitTables {
    std::vector<int32_t> W;
    std::vector<float> H[3];
    std::vector<int> woff, hoff;
};
SplitTables build_split_tables(const HostTables &t, int G, int P);
// positive edge factors as (h, l, exponent, 0): (h 2^30 + l) 2^(exponent - 60)
std::vector<int32_t> fx_edges(const std::vector<double> &e, size_t count);

}  // namespace sfmm
