// FP32 translations (k_translate_fx<float, ...>): the lane layout of the
// 60-bit kernel (sfmm_fx.cuh) on FP32 values.
//
// A translation of order 20 has 800 fused multiply-adds per warp; the former
// layout (both parts of an element in one lane) spent 5 460 instructions on
// it, 660 of them 4-byte table loads, and kept the FP64 pipe busy half of the
// time with a geometry that every thread of a translation repeated.  Here a
// lane holds one part of every (G/2)-th row, so degrees pad to G/2 rows, the
// coefficients of four rows come by one 16-byte load, the geometry is computed
// once per translation, its powers in fixed point and float-float, and the
// target update adds in FP32 (FP64 addition of two FP32 values rounded to FP32
// is the FP32 sum).  The z-translation of M2M and L2L keeps its zero products:
// leaving them out saves fewer FP32 multiply-adds than its shorter loops cost
// (M2M P=20 115 against 146 M/s).  Measured (M2L, one GB300): P=4 763 -> 1 549
// M/s, P=10 341 -> 702, P=20 105 -> 145, P=28 35 -> 52.  What bounds it now:
// the L1 data path, 59% busy with the coefficients (4 bytes per multiply-add
// and lane, whatever the width of the load).
#pragma once

#include "sfmm_fx.cuh"

namespace sfmm {

// a b with subnormal operands and results flushed to zero
__device__ __forceinline__ float mul_ftz(float a, float b)
{
    float r;
    asm("mul.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// fixed-point Q60 value (limbs) to FP32
__device__ __forceinline__ float f32_of_fx(fx v)
{
    const float a = (float)v.h;
    const float b = (float)(v.h - (int)a) + (float)v.l * 0x1p-30f;
    return (a + b) * 0x1p-30f;
}
// (m / 2^60) 2^e as float-float
__device__ __forceinline__ ff ff_of_fxs(long long m, int e)
{
    const fx v = fx_split(m);
    const float a = (float)v.h;
    const float b = (float)(v.h - (int)a) + (float)v.l * 0x1p-30f;
    const float s = pow2f(e - 30);
    return ff_norm(a * s, b * s);
}

template <int ACC>
struct F32Trig {
    float ca[ACC], sa[ACC], cb[ACC], sb[ACC];  // sines signed as in FxTrig
};

// One swap: rows m = r + RS a of W_R (part 0) or W_I (part 1) applied to the
// lane's part; slot t of a degree holds NA/4 float4 per lane, then its last
// NA % 4 rows in one more.
template <int G, int NA>
__device__ __forceinline__ void swap_f32(const float *__restrict__ W, const float *own, int j0, int cnt, int q,
                                         float (&acc)[NA])
{
    constexpr int NQ = (NA + 3) / 4;
    const float *x = own + j0;
    const float *w = W + 4 * q;
#pragma unroll
    for (int a = 0; a < NA; ++a) acc[a] = 0.f;
    auto load = [&](float (&v)[4 * NQ]) {
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            if (NA - 4 * i == 1) {
                v[4 * i] = __ldg(w + 4 * i * G);
            } else if (NA - 4 * i == 2) {
                const float2 u = __ldg(reinterpret_cast<const float2 *>(w + 4 * i * G));
                v[4 * i] = u.x;
                v[4 * i + 1] = u.y;
            } else {
                zvec<float>::get(__ldg(reinterpret_cast<const float4 *>(w + 4 * i * G)), v + 4 * i);
            }
        }
    };
#pragma unroll 2
    for (int t = 0; t < cnt; ++t) {
        const float xv = *x;
        float v[4 * NQ];
        load(v);
        x += 2;
        w += 4 * NQ * G;
#pragma unroll
        for (int a = 0; a < NA; ++a) acc[a] = fmaf(v[a], xv, acc[a]);
    }
}

template <int G, int NA, int ACC>
__device__ __forceinline__ void forward_degree_f32(float *b, int n, const float *__restrict__ W,
                                                   const float *__restrict__ ein, float f, int q,
                                                   const F32Trig<ACC> &tg)
{
    constexpr int RS = G / 2;
    const int d = n + 1, r = q >> 1, part = q & 1, j0 = (r + n + part) & 1, cnt = (d + 1) >> 1;
    float *own = b + n * d + part * d;
    float v[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const bool on = (a + 1 < NA || m < d) && (a || m || !part);  // the imaginary part at m = 0 is zero
        const float x = on ? own[m] : 0.f;
        const float o = __shfl_xor_sync(0xffffffffu, x, 1);
        const float g = f * __ldg(ein + (a + 1 < NA ? m : min(m, n)));
        v[a] = fmaf(g * tg.ca[a], x, g * tg.sa[a] * o);
    }
#pragma unroll
    for (int a = 0; a < NA; ++a)
        if (a + 1 < NA || r + RS * a < d) own[r + RS * a] = v[a];
    __syncwarp();
    swap_f32<G, NA>(W, own, j0, cnt, q, v);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const float o = __shfl_xor_sync(0xffffffffu, v[a], 1);
        const float y = fmaf(tg.cb[a], v[a], tg.sb[a] * o);
        if (a + 1 < NA || r + RS * a < d) own[r + RS * a] = y;
    }
    __syncwarp();
    swap_f32<G, NA>(W, own, j0, cnt, q, v);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a)
        if (a + 1 < NA || r + RS * a < d) own[r + RS * a] = v[a];
    __syncwarp();
}

template <int G, int NA, int ACC>
__device__ __forceinline__ void backward_degree_f32(float *b, int n, const float *__restrict__ W,
                                                    const float *__restrict__ eout, float f, int q,
                                                    const F32Trig<ACC> &tg)
{
    constexpr int RS = G / 2;
    const int d = n + 1, r = q >> 1, part = q & 1, j0 = (r + n + part) & 1, cnt = (d + 1) >> 1;
    float *own = b + n * d + part * d;
    float v[NA];
    swap_f32<G, NA>(W, own, j0, cnt, q, v);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const float o = __shfl_xor_sync(0xffffffffu, v[a], 1);
        const float y = fmaf(tg.cb[a], v[a], -(tg.sb[a] * o));
        if (a + 1 < NA || r + RS * a < d) own[r + RS * a] = y;
    }
    __syncwarp();
    swap_f32<G, NA>(W, own, j0, cnt, q, v);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const float o = __shfl_xor_sync(0xffffffffu, v[a], 1);
        const float g = f * __ldg(eout + (a + 1 < NA ? m : min(m, n)));
        const float y = fmaf(g * tg.ca[a], v[a], -(g * tg.sa[a] * o));
        if (a + 1 < NA || m < d) own[m] = y;
    }
    __syncwarp();
}

}  // namespace sfmm
