// Split precision (k_translate_split): the stages of one translation with the
// swaps and polar rotations in 30-bit block fixed point (sfmm_fixed.cuh) and
// the edges and the z-translation in float-float.  Thread q of a group owns
// the rows m = q + G a, both parts of each.
//
// The kernel is bound by instruction issue on the FP32 and integer pipes, so
// a row block is branch-free (only the last block of a degree has rows past
// it: they compute on zeros and are not stored), the coefficients of two rows
// and both parts come by one 16-byte load, degrees of one block count share a
// loop, and the target update has five loads in flight per lane.  Measured
// (M2L, one GB300): P=10 212 -> 270 M/s, P=12 180 -> 206, P=16 93.1 -> 101.8,
// P=20 51.1 -> 56.5, P=28 15.6 -> 18.0 (8 246 -> 7 626 warp instructions per
// translation at P=16, of which 2 670 float-float arithmetic).  Leaving out the
// zero half of the z-translation of M2M and L2L cost more in its shorter loops
// than it saved (M2M P=16 85.7 against 101.8 M/s).
#pragma once

#include "sfmm_fixed.cuh"
#include "sfmm_fx.cuh"

namespace sfmm {

// Q1.30 cos / sin of m beta for the rotation elements a thread owns
template <int ACC>
struct FixTrig {
    int c[ACC], s[ACC];
};
template <int ACC>
struct FFTrig {
    ff ca[ACC], sa[ACC];
};

// mantissas live in the low word of a buffer slot
__device__ __forceinline__ void st_fixed(float2 *p, int v) { *reinterpret_cast<int *>(p) = v; }

// (a + half) >> s, half = 2^(s-1) (0 for s = 0)
__device__ __forceinline__ int shift_round(long long a, long long half, int s) { return (int)((a + half) >> s); }

// Integer swap of one degree, both parts: rows m = q + G a (a < NA) of the
// Q1.30 matrices applied to the int32 mantissas.  Slot t (column jr + 2t of
// W_R and (jr ^ 1) + 2t of W_I, jr = (q + n) & 1) lies lane by lane: NA/2
// int4 (two rows, W_R and W_I each), then an int2 for an odd last row.
template <int G, int NA>
__device__ __forceinline__ void swap_split(const int2 *__restrict__ W, const float2 *bre, const float2 *bim, int jr,
                                           int cnt, int q, long long (&ar)[NA], long long (&ai)[NA])
{
    constexpr int NP = NA / 2;
    const int *xr = reinterpret_cast<const int *>(bre + jr), *xi = reinterpret_cast<const int *>(bim + (jr ^ 1));
    const int4 *w4 = reinterpret_cast<const int4 *>(W) + q;
    const int2 *w2 = W + 2 * NP * G + q;
#pragma unroll
    for (int a = 0; a < NA; ++a) ar[a] = ai[a] = 0;
    auto load = [&](int2 (&w)[NA]) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int4 u = __ldg(w4 + p * G);
            w[2 * p] = make_int2(u.x, u.y);
            w[2 * p + 1] = make_int2(u.z, u.w);
        }
        if constexpr (NA & 1) w[NA - 1] = __ldg(w2);
    };
    int rn = *xr, in = *xi;
    int2 wn[NA];
    load(wn);
#pragma unroll 4  // 2 loses 3% at P=16
    for (int t = 0; t < cnt; ++t) {  // the next slot's operands load before this one's multiply-adds
        const int vr = rn, vi = in;
        int2 w[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) w[a] = wn[a];
        xr += 4;  // two 8-byte slots
        xi += 4;
        w4 += NA * G / 2;
        w2 += NA * G;
        rn = *xr;
        in = *xi;
        load(wn);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            ar[a] += mul_wide(w[a].x, vr);
            ai[a] += mul_wide(w[a].y, vi);
        }
    }
}

// The two swaps of a degree with the rotation by +beta (SIGN = 1) or -beta
// between them, on mantissas in the buffer at block exponent E; the results in
// (xr, xi) at the exponent returned.
template <int G, int NA, int ACC, int SIGN>
__device__ __forceinline__ int rotate_split(float2 *bre, float2 *bim, int n, const int2 *__restrict__ W, int E, int q,
                                            const FixTrig<ACC> &tq, int (&xr)[NA], int (&xi)[NA])
{
    const int d = n + 1, jr = (q + n) & 1, cnt = (d + 1) >> 1;
    long long ar[NA], ai[NA];
    swap_split<G, NA>(W, bre, bim, jr, cnt, q, ar, ai);
    int sh = group_renorm_shift<G, NA>(ar, ai);
    long long half = (1ll << sh) >> 1;
    E += sh - 30;
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int yr = shift_round(ar[a], half, sh), yi = shift_round(ai[a], half, sh);
        const int c = tq.c[a], s = SIGN * tq.s[a];
        if (a + 1 < NA || q + G * a < d) {
            st_fixed(bre + q + G * a, rot_q30(c, yr, s, yi));
            st_fixed(bim + q + G * a, rot_q30(c, yi, -s, yr));
        }
    }
    __syncwarp();
    swap_split<G, NA>(W, bre, bim, jr, cnt, q, ar, ai);
    sh = group_renorm_shift<G, NA>(ar, ai);
    half = (1ll << sh) >> 1;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        xr[a] = shift_round(ar[a], half, sh);
        xi[a] = shift_round(ai[a], half, sh);
    }
    __syncwarp();
    return E + sh - 30;
}

// float-float rows to mantissas in the buffer; returns the block exponent
template <int G, int NA>
__device__ __forceinline__ int store_fixed_rows(float2 *bre, float2 *bim, int d, int q, const ff (&vr)[NA],
                                                const ff (&vi)[NA])
{
    float mx = 0.f;
#pragma unroll
    for (int a = 0; a < NA; ++a)  // rows past the degree hold zeros
        mx = fmaxf(mx, fmaxf(fabsf(vr[a].hi), fabsf(vi[a].hi)));
    const int E = block_exponent(group_max<G>(mx));
#pragma unroll
    for (int a = 0; a < NA; ++a)
        if (a + 1 < NA || q + G * a < d) {
            st_fixed(bre + q + G * a, ff_to_fixed(vr[a], E));
            st_fixed(bim + q + G * a, ff_to_fixed(vi[a], E));
        }
    __syncwarp();
    return E;
}

// One degree of the forward transform: float-float edge (r-power, basis
// factor, rotation by alpha), then the swaps and the rotation by beta.
template <int G, int NA, int ACC>
__device__ __forceinline__ void forward_degree_split(float2 *b, int n, const int2 *__restrict__ W,
                                                     const ff *__restrict__ ein, ff f, int q, const FFTrig<ACC> &tg,
                                                     const FixTrig<ACC> &tq)
{
    using AR = arith<ff>;
    const int d = n + 1;
    float2 *bre = b + n * d, *bim = bre + d;
    ff vr[NA], vi[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = q + G * a;
        const bool on = a + 1 < NA || m < d;
        const float2 zero = make_float2(0.f, 0.f), ur = on ? bre[m] : zero, ui = on ? bim[m] : zero;
        const ff xr{ur.x, ur.y}, xi{ui.x, ui.y};
        const ff g = AR::mul(f, AR::ldt(ein + (on ? m : n)));
        const ff gc = AR::mul(g, tg.ca[a]), gs = AR::mul(g, tg.sa[a]);
        vr[a] = AR::dot2(gc, xr, AR::neg(gs), xi);
        vi[a] = AR::dot2(gs, xr, gc, xi);
    }
    int E = store_fixed_rows<G, NA>(bre, bim, d, q, vr, vi);
    int xr[NA], xi[NA];
    E = rotate_split<G, NA, ACC, 1>(bre, bim, n, W, E, q, tq, xr, xi);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const ff yr = fixed_to_ff(xr[a], E), yi = fixed_to_ff(xi[a], E);
        if (a + 1 < NA || q + G * a < d) {
            AR::st(bre + q + G * a, yr);
            AR::st(bim + q + G * a, yi);
        }
    }
    __syncwarp();
}

// One degree of the backward transform.
template <int G, int NA, int ACC>
__device__ __forceinline__ void backward_degree_split(float2 *b, int n, const int2 *__restrict__ W,
                                                      const ff *__restrict__ eout, ff f, int q, const FFTrig<ACC> &tg,
                                                      const FixTrig<ACC> &tq)
{
    using AR = arith<ff>;
    const int d = n + 1;
    float2 *bre = b + n * d, *bim = bre + d;
    ff vr[NA], vi[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = q + G * a;
        const bool on = a + 1 < NA || m < d;
        const float2 zero = make_float2(0.f, 0.f), ur = on ? bre[m] : zero, ui = on ? bim[m] : zero;
        vr[a] = ff{ur.x, ur.y};
        vi[a] = ff{ui.x, ui.y};
    }
    int E = store_fixed_rows<G, NA>(bre, bim, d, q, vr, vi);
    int xr[NA], xi[NA];
    E = rotate_split<G, NA, ACC, -1>(bre, bim, n, W, E, q, tq, xr, xi);
#pragma unroll
    for (int a = 0; a < NA; ++a) {  // e^{-i m alpha}, back to the solid basis, r-power scale
        const int m = q + G * a;
        const bool on = a + 1 < NA || m < d;
        const ff ur = fixed_to_ff(xr[a], E), ui = fixed_to_ff(xi[a], E);
        const ff g = AR::mul(f, AR::ldt(eout + (on ? m : n)));
        const ff gc = AR::mul(g, tg.ca[a]), gs = AR::mul(g, tg.sa[a]);
        const ff yr = AR::dot2(gc, ur, gs, ui), yi = AR::dot2(gc, ui, AR::neg(gs), ur);
        if (on) {
            AR::st(bre + m, yr);
            AR::st(bim + m, yi);
        }
    }
    __syncwarp();
}

// blocks [B0, B1) of one z matrix row, pairs of blocks per 16-byte load
template <int G, int B0, int B1, int N>
__device__ __forceinline__ void z_load_ff(const float2 *h, ff (&w)[N])
{
#pragma unroll
    for (int i = B0 / 2; i < (B1 + 1) / 2; ++i) {
        if (B1 - 2 * i == 1) {
            const float2 v = __ldg(h + 2 * i * G);
            w[2 * i] = ff{v.x, v.y};
        } else {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(h + 2 * i * G));
            w[2 * i] = ff{v.x, v.y};
            w[2 * i + 1] = ff{v.z, v.w};
        }
    }
}

// One z-translation column m: outputs n' = m + q + G b (b < NB), both parts.
// H_m lies row by row (input k), pairs of blocks lane by lane, hs entries per
// row.  L2L needs rows k >= n' only: a thread starts at its first (kbeg =
// m + q).
template <int G, int NB>
__device__ __forceinline__ void z_column_split(float2 *b, const float2 *__restrict__ Hm, int hs, int m, int kbeg,
                                               int kend, int nout, int q)
{
    using AR = arith<ff>;
    constexpr int NW = (NB + 1) / 2 * 2;
    ffacc ar[NB], ai[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) ar[i] = ai[i] = AR::acc0();
    if (kbeg < kend) {
        const float2 *h = Hm + (kbeg - m) * hs + 2 * q;
        const float2 *x = b + kbeg * (kbeg + 1) + m;
        ff rn = AR::ld(x), in = AR::ld(x + kbeg + 1), wn[NW];
        z_load_ff<G, 0, NB>(h, wn);
#pragma unroll 2
        for (int k = kbeg; k < kend; ++k) {  // row k+1's operands load before row k's multiply-adds
            const ff vr = rn, vi = in;
            ff w[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) w[i] = wn[i];
            if (k + 1 < kend) {
                x += 2 * (k + 1);
                h += hs;
            }
            rn = AR::ld(x);
            in = AR::ld(x + min(k + 2, kend));
            z_load_ff<G, 0, NB>(h, wn);
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                AR::mac(ar[i], w[i], vr);
                AR::mac(ai[i], w[i], vi);
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int np = m + q + G * i;
        if (np < nout) {
            AR::st(b + np * (np + 1) + m, AR::fin(ar[i]));
            AR::st(b + (np + 1) * (np + 1) + m, AR::fin(ai[i]));
        }
    }
    __syncwarp();
}

}  // namespace sfmm
