// Fused translation kernel: M2M, M2L and L2L over a batch of translations.
//
// One CTA processes tiles of TS translations; each translation is handled by
// a group of G threads that share its working expansion in a per-CTA
// shared-memory buffer.  Per tile:
//
//   1. cooperative, coalesced gather of the TS source expansions into the
//      buffer (solid2buf, microkernel_generic.cpp:341-359),
//   2. per degree n: forward edge (scale r^{-(n+1)} or r^n, rotate e^{i m alpha},
//      change to the orthogonal swap basis), swap, rotate e^{i m beta}, swap
//      (forward_transform_M/L, translations.cpp:37-85 and 190-240),
//   3. z-translation per column m (zm2l / zm2m, translations.cpp:283-296,
//      366-377, 440-451) as a small dense matrix per m,
//   4. per degree n: swap, rotate e^{-i m beta}, swap, backward edge
//      (backward_transform_L/M, translations.cpp:88-187),
//   5. cooperative, coalesced accumulation into the targets (buf2solid,
//      microkernel_generic.cpp:362-380), with FP64/FP32 atomics when
//      targets may repeat.
//
// Thread q of a group owns every G-th (or, holding one part of an element,
// every (G/2)-th) row of a degree and output of a z-translation column; each
// stage keeps its accumulators in registers and reads its inputs from the
// buffer (group members synchronise with __syncwarp).  The number of
// accumulator blocks a stage needs is warp-uniform and selects a stage instance
// compiled for exactly that many blocks, so no block is issued only to be
// predicated off.
// Loop bounds are warp-uniform maxima over the warp's 32/G translations,
// like the reference's lanes padded with zero orders (translations.cpp:504-514);
// inputs past a translation's own order read as zero and outputs past it are
// dropped.
#pragma once

#include <cstdint>
#include <type_traits>

#include "sfmm_arith.cuh"
#include "sfmm_f32.cuh"
#include "sfmm_fx.cuh"
#include "sfmm_split.cuh"
#include "sfmm_params.hpp"

namespace sfmm {

template <class A>
struct src_of {
    using type = double;
};
template <>
struct src_of<float> {
    using type = float;
};


// complex helpers in FP64 for the per-translation geometry
struct cd {
    double c, s;
};
__device__ __forceinline__ cd cmul(cd a, cd b) { return cd{a.c * b.c - a.s * b.s, a.s * b.c + a.c * b.s}; }

__device__ __forceinline__ void prefetch_l2(const void *ptr)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
}

// a table's lines loaded into L1, spread over the CTA's threads
__device__ __forceinline__ void touch_tables(const void *t, int bytes)
{
    for (int o = threadIdx.x * 32; o < bytes; o += blockDim.x * 32) {
        asm volatile("{\n\t.reg .b32 t;\n\tld.global.nc.b32 t, [%0];\n\t}" ::"l"(static_cast<const char *>(t) + o));
    }
}

// Calls f(ic<na>) for na in 1..MAXN (warp-uniform switch).
template <int MAXN, class F>
__device__ __forceinline__ void dispatch(int na, F &&f)
{
    switch (na) {
    case 1: f(ic<1>{}); break;
    case 2: if constexpr (MAXN >= 2) f(ic<2>{}); break;
    case 3: if constexpr (MAXN >= 3) f(ic<3>{}); break;
    case 4: if constexpr (MAXN >= 4) f(ic<4>{}); break;
    case 5: if constexpr (MAXN >= 5) f(ic<5>{}); break;
    case 6: if constexpr (MAXN >= 6) f(ic<6>{}); break;
    case 7: if constexpr (MAXN >= 7) f(ic<7>{}); break;
    case 8: if constexpr (MAXN >= 8) f(ic<8>{}); break;
    default: break;
    }
}

// f(ic<NA>, n) for the degrees n < count in order, NA = ceil((n + 1) / RS):
// RS degrees in a row share an instance, so that no degree pays for a switch.
template <int MAXN, int RS, int NA = 1, class F>
__device__ __forceinline__ void for_degrees(int count, F &&f)
{
#pragma unroll 1
    for (int n = RS * (NA - 1); n < min(RS * NA, count); ++n) f(ic<NA>{}, n);
    if constexpr (NA < MAXN)
        if (RS * NA < count) for_degrees<MAXN, RS, NA + 1>(count, f);
}

// f(ic<NB>, m) for the columns m < mend in order, NB = ceil((nout - m) / RS)
template <int NB, int RS, class F>
__device__ __forceinline__ void for_columns(int m, int mend, int nout, F &&f)
{
#pragma unroll 1
    for (; m < mend && nout - m > RS * (NB - 1); ++m) f(ic<NB>{}, m);
    if constexpr (NB > 1)
        if (m < mend) for_columns<NB - 1, RS>(m, mend, nout, f);
}

// The stages below, down to the geometry, are those of the FP64 kernel for
// orders above 32 (one warp per translation, both parts of an element in one
// lane); the other kernels' are in sfmm_fx.cuh, sfmm_f32.cuh and sfmm_split.cuh.

// Rows of a degree's swap-coefficient block in the instance that runs NA
// accumulator blocks: the tables pad rows to a multiple of 32 above order 32,
// so the row count of every degree served by one instance is the same
// compile-time constant.
template <int G, int NA>
__host__ __device__ constexpr int swap_rows()
{
    return G * NA;
}

// Both swap parts of one degree: rows i = q + G a (a < NA) of W_R applied to
// the real parts (columns j = jr, jr+2, ...) and of W_I to the imaginary
// parts (the complementary checkerboard, columns ji = jr^1, ji+2, ...).
// The coefficient block holds only that checkerboard: slot t of row i is
// column jr(i) + 2t (W_R) or ji(i) + 2t (W_I), and each slot stores the R
// rows of W_R followed by the R rows of W_I, so one pointer walks both with
// compile-time offsets.  Rows are zero-padded to R and slots to (d+3)/2, and
// the buffer slots past each expansion are zero, so every load is
// unconditional; operands of the next column pair are fetched before the
// current pair's multiply-adds (software pipelining), and the real and
// imaginary chains are independent (2*NA accumulations per iteration).
template <class AR, int G, int NA>
__device__ __forceinline__ void swap_both(const typename AR::T *__restrict__ W, const typename AR::Stor *xre,
                                          const typename AR::Stor *xim, int d, int n, int q,
                                          typename AR::Acc (&ar)[NA], typename AR::Acc (&ai)[NA])
{
    using T = typename AR::T;
    constexpr int R = swap_rows<G, NA>();
    const int jr0 = (q + n) & 1, ji0 = jr0 ^ 1;
    const int cnt = (d + 1) >> 1;  // iterations of the longer part
    const T *w = W + q;
    const typename AR::Stor *xr_p = xre + jr0;
    const typename AR::Stor *xi_p = xim + ji0;
    T xrn = AR::ld(xr_p), xin = AR::ld(xi_p);
    T wrn[NA], win[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        wrn[a] = AR::ldt(w + G * a);
        win[a] = AR::ldt(w + R + G * a);
    }
#pragma unroll 1  // the FP64 pipe is the limit
    for (int t = 0; t < cnt; ++t) {
        const T xr = xrn, xi = xin;
        T wr[NA], wi[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            wr[a] = wrn[a];
            wi[a] = win[a];
        }
        xr_p += 2;
        xi_p += 2;
        w += 2 * R;
        xrn = AR::ld(xr_p);
        xin = AR::ld(xi_p);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            wrn[a] = AR::ldt(w + G * a);
            win[a] = AR::ldt(w + R + G * a);
        }
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            AR::mac(ar[a], wr[a], xr);
            AR::mac(ai[a], wi[a], xi);
        }
    }
}

// Per-thread geometry of one translation: e^{i m alpha} and e^{i m beta} for
// the rotation elements m = q + G a this thread owns.
template <class AR, int ACC>
struct Trig {
    typename AR::T ca[ACC], sa[ACC], cb[ACC], sb[ACC];
};

// One degree of the forward transform, NA = ceil(d / G) blocks.
template <class AR, int G, int NA, int ACC>
__device__ __forceinline__ void forward_degree(typename AR::Stor *b, int n,
                                               const typename AR::T *__restrict__ WR,
                                               const typename AR::T *__restrict__ ein, typename AR::T f, int q,
                                               const Trig<AR, ACC> &tg)
{
    using T = typename AR::T;
    using Acc = typename AR::Acc;
    using S = typename AR::Stor;
    const int d = n + 1;
    S *bre = b + n * (n + 1);
    S *bim = b + (n + 1) * (n + 1);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = q + G * a;
        if (m < d) {
            const T xr = AR::ld(bre + m);
            const T xi = AR::ld(bim + m);
            const T g = AR::mul(f, AR::ldt(ein + m));
            const T gc = AR::mul(g, tg.ca[a]), gs = AR::mul(g, tg.sa[a]);
            AR::st(bre + m, AR::dot2(gc, xr, AR::neg(gs), xi));
            AR::st(bim + m, AR::dot2(gs, xr, gc, xi));
        }
    }
    __syncwarp();
#pragma unroll 2
    for (int pass = 0; pass < 2; ++pass) {
        Acc ar[NA], ai[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            ar[a] = AR::acc0();
            ai[a] = AR::acc0();
        }
        swap_both<AR, G, NA>(WR, bre, bim, d, n, q, ar, ai);
        __syncwarp();
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int ii = q + G * a;
            if (ii < d) {
                T vr = AR::fin(ar[a]);
                T vi = AR::fin(ai[a]);
                if (pass == 0) {  // rotation by e^{+i m beta} between the two swaps
                    const T wr = AR::dot2(tg.cb[a], vr, AR::neg(tg.sb[a]), vi);
                    const T wi = AR::dot2(tg.sb[a], vr, tg.cb[a], vi);
                    vr = wr;
                    vi = wi;
                }
                AR::st(bre + ii, vr);
                AR::st(bim + ii, vi);
            }
        }
        __syncwarp();
    }
}

// One degree of the backward transform, NA = ceil(d / G) blocks.
template <class AR, int G, int NA, int ACC>
__device__ __forceinline__ void backward_degree(typename AR::Stor *b, int n,
                                                const typename AR::T *__restrict__ WR,
                                                const typename AR::T *__restrict__ eout, typename AR::T f, int q,
                                                const Trig<AR, ACC> &tg)
{
    using T = typename AR::T;
    using Acc = typename AR::Acc;
    using S = typename AR::Stor;
    const int d = n + 1;
    S *bre = b + n * (n + 1);
    S *bim = b + (n + 1) * (n + 1);
#pragma unroll 2
    for (int pass = 0; pass < 2; ++pass) {
        Acc ar[NA], ai[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            ar[a] = AR::acc0();
            ai[a] = AR::acc0();
        }
        swap_both<AR, G, NA>(WR, bre, bim, d, n, q, ar, ai);
        __syncwarp();
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int ii = q + G * a;
            if (ii < d) {
                T vr = AR::fin(ar[a]);
                T vi = AR::fin(ai[a]);
                if (pass == 0) {  // e^{-i m beta}
                    const T wr = AR::dot2(tg.cb[a], vr, tg.sb[a], vi);
                    const T wi = AR::dot2(tg.cb[a], vi, AR::neg(tg.sb[a]), vr);
                    vr = wr;
                    vi = wi;
                } else {  // e^{-i m alpha}, back to the solid basis, r-power scale
                    const T g = AR::mul(f, AR::ldt(eout + ii));
                    const T gc = AR::mul(g, tg.ca[a]), gs = AR::mul(g, tg.sa[a]);
                    const T wr = AR::dot2(gc, vr, gs, vi);
                    const T wi = AR::dot2(gc, vi, AR::neg(gs), vr);
                    vr = wr;
                    vi = wi;
                }
                AR::st(bre + ii, vr);
                AR::st(bim + ii, vi);
            }
        }
        __syncwarp();
    }
}

// One z-translation column m, outputs n' = m + q + G a (a < NA), kept where
// n' < nout: out(n',m) = sum_{k=kbeg}^{kend-1} H_m[k-m][n'-m] in(k,m), in
// place.  H_m's output rows are zero-padded to a multiple of 8 (HR), so the
// coefficient loads need no bounds check.
template <class AR, int G, int NA>
__device__ __forceinline__ void z_column(typename AR::Stor *b, const typename AR::T *__restrict__ Hm, int HR, int m,
                                         int kbeg, int kend, int nout, int q)
{
    using T = typename AR::T;
    using Acc = typename AR::Acc;
    Acc ar[NA], ai[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        ar[a] = AR::acc0();
        ai[a] = AR::acc0();
    }
    if (kbeg < kend) {
        // row k of column m: real part at ro = k(k+1) + m, imaginary part at
        // ro + k + 1; both advance by 2(k+1) per row
        const T *h_p = Hm + (long long)(kbeg - m) * HR + q;
        int ro = kbeg * (kbeg + 1) + m, step = 2 * (kbeg + 1);
        T xr = AR::ld(b + ro), xi = AR::ld(b + ro + kbeg + 1);
        T hc[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) hc[a] = AR::ldt(h_p + G * a);
#pragma unroll 2
        for (int k = kbeg; k < kend - 1; ++k) {  // the operands of row k+1 load before row k's multiply-adds
            ro += step;
            step += 2;
            h_p += HR;
            const T xrn = AR::ld(b + ro), xin = AR::ld(b + ro + k + 2);
            T hn[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) hn[a] = AR::ldt(h_p + G * a);
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                AR::mac(ar[a], hc[a], xr);
                AR::mac(ai[a], hc[a], xi);
            }
            xr = xrn;
            xi = xin;
#pragma unroll
            for (int a = 0; a < NA; ++a) hc[a] = hn[a];
        }
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            AR::mac(ar[a], hc[a], xr);
            AR::mac(ai[a], hc[a], xi);
        }
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int np = m + q + G * a;
        if (np < nout) {
            AR::st(b + np * (np + 1) + m, AR::fin(ar[a]));
            AR::st(b + (np + 1) * (np + 1) + m, AR::fin(ai[a]));
        }
    }
    __syncwarp();
}

// e^{i q gamma} by binary powers of e^{i gamma}, then steps of e^{i G gamma}:
// the rotation factors of the elements m = q + G a a thread owns.
template <int G, int ACC, class C, class Mul, class Out>
__device__ __forceinline__ void rotation_powers(C ea, C eb, C one, int q, Mul cmul_, Out out)
{
    C pa = one, pb = one, ka = ea, kb = eb;
#pragma unroll
    for (int bit = 1; bit < G; bit <<= 1) {
        if (q & bit) {
            pa = cmul_(pa, ka);
            pb = cmul_(pb, kb);
        }
        ka = cmul_(ka, ka);
        kb = cmul_(kb, kb);
    }
#pragma unroll
    for (int a = 0; a < ACC; ++a) {
        out(a, pa, pb);
        if (a + 1 < ACC) {
            pa = cmul_(pa, ka);
            pb = cmul_(pb, kb);
        }
    }
}

struct cff {
    ff c, s;
};

// Degree n of every coefficient index c below kDegreeTableSize (n(n+1) <= c
// < (n+1)(n+2)): the FP32-range kernels scale each coefficient by a power of
// two per degree in the gather and the target update, and one cached byte
// load per coefficient issues fewer instructions than computing the degree.
// Covers the buffers of every order those kernels run (up to 28: at most
// 28 * 29 + 4 slots plus padding), checked on the host against
// kDegreeTableSize.
struct DegreeTable {
    unsigned char d[kDegreeTableSize];
};
constexpr DegreeTable make_degree_table()
{
    DegreeTable t{};
    int n = 0;
    for (int c = 0; c < kDegreeTableSize; ++c) {
        while ((n + 1) * (n + 2) <= c) ++n;
        t.d[c] = (unsigned char)n;
    }
    return t;
}
__device__ const DegreeTable kDegree = make_degree_table();
__device__ __forceinline__ int degree_at(int c) { return (int)__ldg(kDegree.d + c); }

// source coefficient times 2^e in the arithmetic's storage type (exact)
__device__ __forceinline__ ff src_scaled(double x, int e, const ff *) { return ff_from_d_scaled0(x, e); }
__device__ __forceinline__ float src_scaled(float x, int e, const float *) { return f_scaled(x, e); }

// Per-thread geometry of one translation in FP64 (orders above 32): |shift|,
// its inverse and the rotation factors.
template <class AR, int G, int ACC>
struct Geometry {
    double r, rinv;
    Trig<AR, ACC> tg;

    __device__ __forceinline__ Geometry(double x, double y, double z, int q)
    {
        const double rxy = hypot(x, y);
        r = hypot(rxy, z);
        rinv = 1.0 / r;
        const cd ea = (rxy == 0) ? cd{1.0, 0.0} : cd{y / rxy, x / rxy};
        const cd eb = cd{z * rinv, -rxy * rinv};
        rotation_powers<G, ACC>(ea, eb, cd{1.0, 0.0}, q, [](cd a, cd b) { return cmul(a, b); },
                                [&](int a, cd pa, cd pb) {
                                    tg.ca[a] = pa.c;
                                    tg.sa[a] = pa.s;
                                    tg.cb[a] = pb.c;
                                    tg.sb[a] = pb.s;
                                });
    }
};

// The same in float-float for the split kernel, which executes no FP64
// instruction here (GB300's FP64 pipe runs at 1/64 of the FP32 rate).
template <int G, int ACC>
struct SplitGeometry {
    ff r, rinv;
    FFTrig<ACC> tg;
    FixTrig<ACC> tq;

    __device__ __forceinline__ SplitGeometry(double x, double y, double z, int q)
    {
        using A = arith<ff>;
        const ff fz = ff_from_d_int(z);
        const ff_transverse t = ff_transverse_of(x, y);
        r = ff_sqrt(A::add(t.r2, A::mul(fz, fz)));
        rinv = ff_rcp(r);
        const cff ea{t.c, t.s};
        const cff eb{A::mul(fz, rinv), A::neg(A::mul(t.r, rinv))};
        auto cm = [](cff a, cff b) {
            return cff{A::dot2(a.c, b.c, A::neg(a.s), b.s), A::dot2(a.s, b.c, a.c, b.s)};
        };
        rotation_powers<G, ACC>(ea, eb, cff{ff{1.f, 0.f}, ff{0.f, 0.f}}, q, cm, [&](int a, cff pa, cff pb) {
            tg.ca[a] = pa.c;
            tg.sa[a] = pa.s;
            // Q1.30
            tq.c[a] = __float2int_rn(pb.c.hi * 1073741824.f) + __float2int_rn(pb.c.lo * 1073741824.f);
            tq.s[a] = __float2int_rn(pb.s.hi * 1073741824.f) + __float2int_rn(pb.s.lo * 1073741824.f);
        });
    }
};

// FIX selects block fixed-point swaps and beta rotations (float-float only).
// HBM: expansions in device memory (L2 prefetch and a 4x unrolled gather);
// false for host memory read over the link, where both cost end-to-end rate.
// WORK: tiles come from a work list (persistent launches of fused plans)
// instead of a fixed stride over the batch.
template <class A, int G, int ACC, bool FIX, bool HBM, bool WORK>
__device__ __forceinline__ void translate_body(const KParams &p)
{
    using AR = arith<A>;
    using T = typename AR::T;
    using S = typename AR::Stor;
    using Src = typename src_of<A>::type;
    static_assert(sizeof(S) == sizeof(Src), "buffer slots hold one source value");
    static_assert(32 % G == 0, "a translation's threads must share a warp");
    // FIX: the float-float kernel with 30-bit block fixed-point swaps, or the
    // kernels whose lanes hold one part of an element each (PL): FP64 in
    // 60-bit block fixed point, and FP32
    constexpr bool PL = FIX && !AR::split;
    constexpr bool F32 = std::is_same<A, float>::value;

    // loads in flight per lane in the source gather and the target update
    // (M2L P=16 x 10^6, split: 8 and 4 over 4 and 1 are worth 2.2%)
    // FP32-range arithmetics run every translation at the length scale of
    // its shift: lambda = 2^ks with |shift| / lambda in [2, 7), sources (and
    // the shift) divided by lambda^n (multipoles) or lambda^-(n+1) (locals),
    // results multiplied back -- the operators are homogeneous, and powers of
    // two are exact, so only the range changes.  With r = |shift| / lambda in
    // [2, 7) the edge factors (r^-(n+1) or r^n times the basis factors
    // sqrt((n-m)!(n+m)!) or their inverses, up to 5e35 at order 28) stay
    // inside the FP32 range at every geometry scale; shifts whose largest
    // component lies in [2, 4) run unscaled
    constexpr bool kScale = !std::is_same<A, double>::value;
    constexpr int kGatherUnroll = FIX ? 8 : 4;
    constexpr int kAccBatch = 5;

    extern __shared__ __align__(16) unsigned char smem[];
    const int TS = p.TS;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int q = tid % G;
    const int slot = tid / G;
    const int P = p.P;
    const unsigned FULL = 0xffffffffu;

    S *buf0 = reinterpret_cast<S *>(smem);
    FxGeo *geo = reinterpret_cast<FxGeo *>(smem + (size_t)TS * p.spad * sizeof(S));  // PL only
    uint32_t *meta = reinterpret_cast<uint32_t *>(smem + (size_t)TS * p.spad * sizeof(S) + (PL ? TS * sizeof(FxGeo) : 0));
    uint32_t *m_sidx = meta;
    uint32_t *m_tidx = meta + TS;
    uint32_t *m_pin = meta + 2 * TS;
    uint32_t *m_pout = meta + 3 * TS;
    uint32_t *m_id = meta + 4 * TS;

    const T *W = reinterpret_cast<const T *>(p.W);
    const T *EIN = reinterpret_cast<const T *>(p.ein);
    const T *EOUT = reinterpret_cast<const T *>(p.eout);
    const T *H = reinterpret_cast<const T *>(p.H);
    const Src *src = reinterpret_cast<const Src *>(p.src);
    Src *dst = reinterpret_cast<Src *>(p.dst);
    const int op = p.op;
    if constexpr (FIX) {
        // this order's tables into L1, all loads in flight at once (the
        // transforms would meet them one miss after the other)
        touch_tables(p.W, p.wbytes);
        touch_tables(p.H, p.hbytes);
        constexpr int kEdge = F32 ? 4 : AR::split ? 8 : 16;
        touch_tables(p.ein, P * (P + 1) / 2 * kEdge);
        touch_tables(p.eout, P * (P + 1) / 2 * kEdge);
    }

    for (long long tile = blockIdx.x;; tile += gridDim.x) {
        // this tile's range of the processing order: a fixed stride over the
        // batch, or the next entry of the work list (its two words after the
        // meta arrays: work-list launches carry 8 more bytes of shared memory)
        long long base = tile * TS;
        int cnt = TS;
        if constexpr (WORK) {
            uint32_t *wsh = meta + 5 * TS;
            if (tid == 0) {
                const unsigned w = atomicAdd(p.work_counter, 1u);
                const uint2 d = w < (unsigned long long)p.nwork ? p.work[w] : make_uint2(0u, 0xffffffffu);
                wsh[0] = d.x;
                wsh[1] = d.y;
            }
            __syncthreads();
            if (wsh[1] == 0xffffffffu) break;
            base = wsh[0];
            cnt = (int)wsh[1];
        } else if (base >= p.n) {
            break;
        }
        const long long i = base + slot;
        bool valid = i < p.n;
        if constexpr (WORK) valid = valid && slot < cnt;
        uint32_t t = 0, si = 0, ti = 0;
        if (valid) t = p.perm ? p.perm[i] : (uint32_t)i;
        int pin = 0, pout = 0;
        double x = 0, y = 0, z = 1;
        if (valid && t < p.nidx) {  // one round of independent loads
            si = p.sidx ? p.sidx[t] : t;
            ti = p.tidx ? p.tidx[t] : t;
            pin = (int)p.pin[t];
            pout = (int)p.pout[t];
            x = p.shift[3 * (long long)t];
            y = p.shift[3 * (long long)t + 1];
            z = p.shift[3 * (long long)t + 2];
        }
        // malformed entries (the unchecked API's undefined behaviour) are
        // skipped and reported instead of touching memory out of bounds
        if (valid && (t >= p.nidx || si >= p.nsrc || ti >= p.ndst || pin > P || pout > P || pin < 0 || pout < 0)) {
            if (q == 0) atomicOr(p.status, 1);
            valid = false;
            pin = pout = 0;
            x = y = 0;
            z = 1;
        }
        if (op == OP_M2M) {  // M2M translates by the negated shift (translations.cpp:331-333)
            x = -x;
            y = -y;
            z = -z;
        }
        const bool ident = valid && op != OP_M2L && (x * x + y * y + z * z) == 0.0;
        int ident_p = 0;
        if (ident) {  // zero shift: direct prefix add (translations.cpp:540-547)
            ident_p = min(pin, pout);
            pin = 0;
            pout = 0;
            x = 0;
            y = 0;
            z = 1;
        }
        if (op == OP_L2L) pout = min(pin, pout);  // output degrees >= P_in receive nothing (translations.cpp:412)
        int ks = 0;
        if constexpr (kScale) {
            const int e3 = max(exp_of(x), max(exp_of(y), exp_of(z)));  // |shift| in [2^e3, sqrt(3) 2^(e3+1))
            if (valid && !ident && e3 > -(1 << 19)) {
                ks = e3 - 1;
                x = d_scaled(x, -ks);
                y = d_scaled(y, -ks);
                z = d_scaled(z, -ks);
            }
        }
        if (q == 0) {
            m_sidx[slot] = valid ? si : 0;
            m_tidx[slot] = valid ? ti : 0;
            m_pin[slot] = (uint32_t)pin | ((uint32_t)(ks + 32768) << 16);  // order, and the scale above it
            m_pout[slot] = pout;
            m_id[slot] = ident_p;
            if constexpr (PL) *reinterpret_cast<double3 *>(geo + slot) = make_double3(x, y, z);
        }
        __syncthreads();
        if constexpr (PL) {  // one thread per translation: the others' lanes would only repeat it
            if (tid < TS) {
                const double3 v = *reinterpret_cast<const double3 *>(geo + tid);
                fx_geometry(v.x, v.y, v.z, geo + tid);
            }
        }

        // 1. gather sources into the buffer (one warp per expansion, lanes over
        //    coefficients) in the arithmetic's storage format, zero past each
        //    source's order and in the padding (the swap loops read a few
        //    slots past a row and multiply them by zero coefficients).
        //    Sources and targets stream through with evict-first hints so the
        //    coefficient tables stay in the L1 left beside the buffers.
        [[maybe_unused]] unsigned low = 0xffffffffu;
        for (int s = warp; s < TS; s += nwarps) {
            const int ps = (int)(m_pin[s] & 0xffffu);
            const int cnt = ps * (ps + 1);
            const Src *sp = p.src_ptr ? reinterpret_cast<const Src *>(p.src_ptr[m_sidx[s]])
                                      : src + (long long)m_sidx[s] * p.sstride;
            S *bp = buf0 + (long long)s * p.spad;
            if constexpr (kScale) {  // coefficient c of degree n times lambda^-n or lambda^(n+1)
                const int ksg = (int)(m_pin[s] >> 16) - 32768;
                const int es = op == OP_L2L ? ksg : -ksg;  // per degree
                const int e0 = op == OP_L2L ? ksg : 0;
                if constexpr (F32) {
                    // every factor an FP32 normal: a product does it, with
                    // subnormals flushed as f_scaled does
                    if (abs(es) * P + abs(e0) <= 126) {
#pragma unroll(kGatherUnroll)
                        for (int c = lane; c < p.spad; c += 32)
                            bp[c] = c < cnt ? mul_ftz(__ldcs(sp + c), pow2f(es * degree_at(c) + e0)) : 0.f;
                        continue;
                    }
                }
#pragma unroll(kGatherUnroll)
                for (int c = lane; c < p.spad; c += 32)
                    AR::st(bp + c, c < cnt ? src_scaled(__ldcs(sp + c), es * degree_at(c) + e0, (const T *)nullptr)
                                           : AR::zero());
            } else {
                auto put = [&](int c) {
                    const Src v = c < cnt ? __ldcs(sp + c) : Src(0);
                    if constexpr (PL && !F32) low = fx_low(v, low);
                    AR::st(bp + c, AR::from_src(v));
                };
                if constexpr (HBM) {  // kGatherUnroll loads in flight per lane
#pragma unroll(kGatherUnroll)
                    for (int c = lane; c < p.spad; c += 32) put(c);
                } else {
                    for (int c = lane; c < p.spad; c += 32) put(c);
                }
            }
        }
        if constexpr (PL && !F32)
            if (__any_sync(FULL, fx_tiny(low)))
#pragma unroll 1
                for (int s = warp; s < TS; s += nwarps)
                    fx_raise_rows(buf0 + (long long)s * p.spad, p.spad, (int)(m_pin[s] & 0xffffu), lane);
        __syncthreads();

        // L2 prefetch, spread over the group: this tile's targets (read at the
        // end of the tile) and the next tile's sources (read at its start),
        // so that both phases meet L2 instead of DRAM.  Device arrays only;
        // every address lies inside an expansion the entry may touch.
        if (HBM && !WORK && !p.src_ptr) {
            const int tc = max(pout * (pout + 1), ident_p * (ident_p + 1));
            if (valid && tc) {
                const char *dp = reinterpret_cast<const char *>(dst + (long long)ti * p.dstride);
                for (int o = q * 128; o < tc * (int)sizeof(Src); o += G * 128) prefetch_l2(dp + o);
            }
            const long long i2 = (tile + gridDim.x) * TS + slot;
            if (i2 < p.n) {
                const uint32_t t2 = p.perm ? p.perm[i2] : (uint32_t)i2;
                if (t2 < p.nidx) {
                    const uint32_t s2 = p.sidx ? p.sidx[t2] : t2;
                    const int pin2 = (int)p.pin[t2];
                    if (s2 < p.nsrc && pin2 > 0 && pin2 <= P) {
                        const char *sp2 = reinterpret_cast<const char *>(src + (long long)s2 * p.sstride);
                        for (int o = q * 128; o < pin2 * (pin2 + 1) * (int)sizeof(Src); o += G * 128)
                            prefetch_l2(sp2 + o);
                    }
                }
            }
        }

        S *b = buf0 + (long long)slot * p.spad;
        int pin_w = __reduce_max_sync(FULL, pin);
        int pout_w = __reduce_max_sync(FULL, pout);
        // A tile of more than one pair of orders runs all its warps to the
        // tile's largest: they wait for each other at its end anyway, and in
        // step they share the instruction cache, which holds a part of the
        // FP64 kernel's unrolled rows only (translations of random orders in
        // one launch, M2L: 2 to 10 161 -> 220 M/s, 4 to 16 58 -> 82).  Slots
        // without a translation, and zero shifts, have no orders, and a warp
        // of them alone does nothing.  Each warp finds this out for itself: a
        // vote of the CTA at the barrier above cost the registers of a flag
        // (spills at orders 5 to 24; FMM pass at P=12 36.5 ms, 31.7 now).
        if constexpr (PL && !F32) {
            static_assert(kFxThreads / 4 <= 32, "a lane per translation of the tile");
            const unsigned o = lane < TS ? (m_pin[lane] & 0xffffu) | m_pout[lane] << 16 : 0u;
            const unsigned some = __ballot_sync(FULL, o != 0u);
            const unsigned first = __shfl_sync(FULL, o, some ? __ffs(some) - 1 : 0);
            if ((pin_w | pout_w) && __any_sync(FULL, o != 0u && o != first)) {
                pin_w = __reduce_max_sync(FULL, o & 0xffffu);
                pout_w = __reduce_max_sync(FULL, o >> 16);
            }
        }

        if constexpr (PL && F32) {
            const FxGeo &ge = geo[slot];
            const int part = q & 1;
            F32Trig<ACC> tg;
            {
                fx c[ACC], sn[ACC];
                fx_powers<G / 2, ACC>(ge.ca, ge.sa, q >> 1, part, c, sn);
#pragma unroll
                for (int a = 0; a < ACC; ++a) {
                    tg.ca[a] = f32_of_fx(c[a]);
                    tg.sa[a] = f32_of_fx(sn[a]);
                }
                fx_powers<G / 2, ACC>(ge.cb, ge.sb, q >> 1, part, c, sn);
#pragma unroll
                for (int a = 0; a < ACC; ++a) {
                    tg.cb[a] = f32_of_fx(c[a]);
                    tg.sb[a] = f32_of_fx(sn[a]);
                }
            }
            // the scaled |shift| lies in [2, 7); not finite or zero: NaN
            const bool bad = ge.re == kFxBad;
            const ff nan{__int_as_float(0x7fffffff), 0.f}, one{1.f, 0.f};
            const ff r = bad ? nan : ff_of_fxs(ge.r, ge.re), rinv = bad ? nan : ff_of_fxs(ge.rinv, ge.rinve);
            // 2. forward transforms: r^n (L input) or r^-(n+1) (M input)
            ff f = op == OP_L2L ? (bad ? nan : one) : rinv;
            const ff fstep = op == OP_L2L ? r : rinv;
            const T *w = W, *e = EIN;
            for_degrees<ACC, G / 2>(pin_w, [&](auto na, int n) {
                constexpr int NA = decltype(na)::value;
                forward_degree_f32<G, NA, ACC>(b, n, w, e, f.hi, q, tg);
                w += ((n + 2) >> 1) * ((NA + 3) / 4 * 4 * G);
                e += n + 1;
                f = ff_mul(f, fstep);
            });
            // 3. z-translation (columns m >= min(P_in, P_out) of the outputs
            // stay zero: their rows beyond P_in were zero-filled by the gather)
            const T *h = H;
            for_columns<ACC, G / 2>(0, min(pin_w, pout_w), pout_w, [&](auto nb, int m) {
                const int hs = fx_hrow(p.Ptab - m, G, 4);
                z_column_part<float, G, decltype(nb)::value>(b, h, hs, m, op == OP_M2M ? min(pin_w, pout_w) : pin_w, pout_w, q);
                h += (p.Ptab - m) * hs;
            });
            // 4. backward transforms: r^(n+1) (M output) or r^-n (L output)
            f = op == OP_M2M ? r : one;
            const ff bstep = op == OP_M2M ? r : rinv;
            w = W;
            e = EOUT;
            for_degrees<ACC, G / 2>(pout_w, [&](auto na, int n) {
                constexpr int NA = decltype(na)::value;
                backward_degree_f32<G, NA, ACC>(b, n, w, e, f.hi, q, tg);
                w += ((n + 2) >> 1) * ((NA + 3) / 4 * 4 * G);
                e += n + 1;
                f = ff_mul(f, bstep);
            });
        } else if constexpr (PL) {
            const FxGeo &ge = geo[slot];
            const int part = q & 1;
            FxTrig<ACC> tg;
            fx_powers<G / 2, ACC>(ge.ca, ge.sa, q >> 1, part, tg.ca, tg.sa);
            fx_powers<G / 2, ACC>(ge.cb, ge.sb, q >> 1, part, tg.cb, tg.sb);
            const fxs r{fx_split(ge.r), ge.re}, rinv{fx_split(ge.rinv), ge.rinve}, one{fx{1 << 29, 0}, 1};
            const bool bad = ge.re == kFxBad;
            const int2 *W = reinterpret_cast<const int2 *>(p.W);
            const int4 *EIN = reinterpret_cast<const int4 *>(p.ein), *EOUT = reinterpret_cast<const int4 *>(p.eout);
            const double *H = reinterpret_cast<const double *>(p.H);
            // 2. forward transforms: r^n (L input) or r^-(n+1) (M input)
            fxs f = op == OP_L2L ? one : rinv;
            const fxs fstep = op == OP_L2L ? r : rinv;
            const int2 *w = W;
            const int4 *e = EIN;
            for_degrees<ACC, G / 2>(pin_w, [&](auto na, int n) {
                constexpr int NA = decltype(na)::value;
                forward_degree_fx<G, NA, ACC>(b, n, w, e, f, bad, p.spad, q, tg);
                w += ((n + 2) >> 1) * (NA * G);
                e += n + 1;
                f = fxs_mul(f, fstep);
            });
            // 3. z-translation (columns m >= min(P_in, P_out) of the outputs
            // stay zero: their rows beyond P_in were zero-filled by the gather)
            const double *h = H;
            for_columns<ACC, G / 2>(0, min(pin_w, pout_w), pout_w, [&](auto nb, int m) {
                const int hs = fx_hrow(p.Ptab - m, G);
                z_column_op<double, G, decltype(nb)::value>(op, b, h, hs, m, pin_w, pout_w, q);
                h += (p.Ptab - m) * hs;
            });
            // 4. backward transforms: r^(n+1) (M output) or r^-n (L output)
            f = op == OP_M2M ? r : one;
            const fxs bstep = op == OP_M2M ? r : rinv;
            w = W;
            e = EOUT;
            for_degrees<ACC, G / 2>(pout_w, [&](auto na, int n) {
                constexpr int NA = decltype(na)::value;
                backward_degree_fx<G, NA, ACC>(b, n, w, e, f, bad, q, tg);
                w += ((n + 2) >> 1) * (NA * G);
                e += n + 1;
                f = fxs_mul(f, bstep);
            });
        } else if constexpr (AR::split) {
            const SplitGeometry<G, ACC> geo(x, y, z, q);
            // 2. forward transforms: r^n (L input) or r^-(n+1) (M input), by
            // repeated multiplication (error ~n 2^-48)
            const ff one{1.f, 0.f};
            ff f = op == OP_L2L ? one : geo.rinv;
            const ff fstep = op == OP_L2L ? geo.r : geo.rinv;
            const int2 *w = reinterpret_cast<const int2 *>(p.W);
            const T *e = EIN;
            for_degrees<ACC, G>(pin_w, [&](auto na, int n) {
                constexpr int NA = decltype(na)::value;
                forward_degree_split<G, NA, ACC>(b, n, w, e, f, q, geo.tg, geo.tq);
                w += ((n + 2) >> 1) * (NA * G);
                e += n + 1;
                f = ff_mul(f, fstep);
            });
            // 3. z-translation (columns m >= min(P_in, P_out) of the outputs
            // stay zero: their rows beyond P_in were zero-filled by the gather)
            const float2 *h = reinterpret_cast<const float2 *>(p.H);
            for_columns<ACC, G>(0, min(pin_w, pout_w), pout_w, [&](auto nb, int m) {
                const int hs = fx_hrow(p.Ptab - m, 2 * G);
                z_column_split<G, decltype(nb)::value>(b, h, hs, m, op == OP_L2L ? m + q : m,
                                                       op == OP_M2M ? min(pin_w, pout_w) : pin_w, pout_w, q);
                h += (p.Ptab - m) * hs;
            });
            // 4. backward transforms: r^(n+1) (M output) or r^-n (L output)
            f = op == OP_M2M ? geo.r : one;
            const ff bstep = op == OP_M2M ? geo.r : geo.rinv;
            w = reinterpret_cast<const int2 *>(p.W);
            e = EOUT;
            for_degrees<ACC, G>(pout_w, [&](auto na, int n) {
                constexpr int NA = decltype(na)::value;
                backward_degree_split<G, NA, ACC>(b, n, w, e, f, q, geo.tg, geo.tq);
                w += ((n + 2) >> 1) * (NA * G);
                e += n + 1;
                f = ff_mul(f, bstep);
            });
        } else {
            // geometry (euler, microkernel_generic.cpp:37-97)
            const Geometry<AR, G, ACC> geo(x, y, z, q);
            // 2. forward transforms, degree by degree; r-power scale of degree
            // n: r^n (L input) or r^-(n+1) (M input)
            T f = op == OP_L2L ? 1.0 : geo.rinv;
            const T fstep = op == OP_L2L ? geo.r : geo.rinv;
            for (int n = 0; n < pin_w; ++n) {
                const T *WR = W + __ldg(p.woff + n);
                dispatch<ACC>((n + G) / G, [&](auto na) {
                    forward_degree<AR, G, decltype(na)::value, ACC>(b, n, WR, EIN + n * (n + 1) / 2, f, q, geo.tg);
                });
                f *= fstep;
            }
            // 3. z-translation, column by column.  Columns m >= min(P_in, P_out)
            //    of the outputs stay zero (trans2swap_buf, microkernel_generic.cpp:308-338):
            //    their rows beyond P_in were zero-filled by the gather.
            const int mend = min(pin_w, pout_w);
            for (int m = 0; m < mend; ++m) {
                const int HR = (p.Ptab - m + p.rowpad - 1) & ~(p.rowpad - 1);
                const T *Hm = H + __ldg(p.hoff + m);
                // M2M only needs inputs k <= n' and L2L only k >= n'
                const int kbeg = (op == OP_L2L) ? m + q : m;
                const int kend = (op == OP_M2M) ? mend : pin_w;
                dispatch<ACC>((pout_w - m + G - 1) / G, [&](auto na) {
                    z_column<AR, G, decltype(na)::value>(b, Hm, HR, m, kbeg, kend, pout_w, q);
                });
            }
            // 4. backward transforms
            f = op == OP_M2M ? geo.r : 1.0;  // r^(n+1) (M output) or r^-n (L output)
            const T bstep = op == OP_M2M ? geo.r : geo.rinv;
            for (int n = 0; n < pout_w; ++n) {
                const T *WR = W + __ldg(p.woff + n);
                dispatch<ACC>((n + G) / G, [&](auto na) {
                    backward_degree<AR, G, decltype(na)::value, ACC>(b, n, WR, EOUT + n * (n + 1) / 2, f, q, geo.tg);
                });
                f *= bstep;
            }
        }
        __syncthreads();

        // 5. accumulate into the targets (one warp per expansion)
        for (int s = warp; s < TS; s += nwarps) {
            const int po = (int)m_pout[s];
            const int pid = (int)m_id[s];
            const int cnt = max(po * (po + 1), pid * (pid + 1));
            if (!cnt) continue;
            const S *bp = buf0 + (long long)s * p.spad;
            const Src *sp = p.src_ptr ? reinterpret_cast<const Src *>(p.src_ptr[m_sidx[s]])
                                      : src + (long long)m_sidx[s] * p.sstride;
            Src *dp = p.dst_ptr ? reinterpret_cast<Src *>(p.dst_ptr[m_tidx[s]]) : dst + (long long)m_tidx[s] * p.dstride;
            // back from the translation's length scale: output coefficient c of
            // degree j times lambda^j (multipoles) or lambda^-(j+1) (locals)
            const int ksa = (int)(m_pin[s] >> 16) - 32768;
            const int eo = op == OP_M2M ? ksa : -ksa, eo0 = op == OP_M2M ? 0 : -ksa;
            if constexpr (PL && F32) {
                // the FP32 sum equals the FP64 sum rounded to FP32
                if (!pid && abs(eo) * P + abs(eo0) <= 126) {
                    for (int c0 = lane; c0 < cnt; c0 += 32 * kAccBatch) {
                        float v[kAccBatch];
                        if (!p.atomic) {
#pragma unroll
                            for (int u = 0; u < kAccBatch; ++u) v[u] = c0 + 32 * u < cnt ? __ldcs(dp + c0 + 32 * u) : 0.f;
                        }
#pragma unroll
                        for (int u = 0; u < kAccBatch; ++u) {
                            const int c = c0 + 32 * u;
                            if (c >= cnt) continue;
                            const float y = bp[c] * pow2f(eo * degree_at(c) + eo0);
                            if (p.atomic) atomicAdd(dp + c, y);
                            else __stcs(dp + c, v[u] + y);
                        }
                    }
                    continue;
                }
            } else if constexpr (PL) {
                // kAccBatch target loads in flight per lane
                if (!p.atomic && !pid) {
                    for (int c0 = lane; c0 < cnt; c0 += 32 * kAccBatch) {
                        double v[kAccBatch];
#pragma unroll
                        for (int u = 0; u < kAccBatch; ++u) v[u] = c0 + 32 * u < cnt ? __ldcs(dp + c0 + 32 * u) : 0.0;
#pragma unroll
                        for (int u = 0; u < kAccBatch; ++u)
                            if (c0 + 32 * u < cnt) __stcs(dp + c0 + 32 * u, v[u] + bp[c0 + 32 * u]);
                    }
                    continue;
                }
            }
            if constexpr (AR::split) {
                // kAccBatch target loads in flight per lane; hi and lo widen by
                // exponent re-biasing; two FP64 additions
                if (!pid) {
                    for (int c0 = lane; c0 < cnt; c0 += 32 * kAccBatch) {
                        double v[kAccBatch];
                        if (!p.atomic) {
#pragma unroll
                            for (int u = 0; u < kAccBatch; ++u) v[u] = c0 + 32 * u < cnt ? __ldcs(dp + c0 + 32 * u) : 0.0;
                        }
#pragma unroll
                        for (int u = 0; u < kAccBatch; ++u) {
                            const int c = c0 + 32 * u;
                            if (c >= cnt) continue;
                            const T t = AR::ld(bp + c);
                            const int e = eo * degree_at(c) + eo0;
                            const double hd = d_from_f_scaled(t.hi, e), lo = d_from_f_scaled(t.lo, e);
                            if (p.atomic) atomicAdd(dp + c, hd + lo);
                            else __stcs(dp + c, (v[u] + hd) + lo);
                        }
                    }
                    continue;
                }
            }
            for (int c = lane; c < cnt; c += 32) {
                const int j = kScale ? degree_at(c) : 0;
                if constexpr (AR::split) {
                    // hi and lo widen by exponent re-biasing; two FP64 additions
                    // (one FP64 addition after an integer-only hi + lo measured
                    // 2% slower: the kernel is issue bound, not FP64 bound)
                    double v = p.atomic ? 0.0 : (double)__ldcs(dp + c);
                    if (c < po * (po + 1)) {
                        const T t = AR::ld(bp + c);
                        const int e = eo * j + eo0;
                        const double hd = d_from_f_scaled(t.hi, e), lo = d_from_f_scaled(t.lo, e);
                        v = p.atomic ? hd + lo : (v + hd) + lo;
                    }
                    if (c < pid * (pid + 1)) v += (double)__ldcs(sp + c);
                    if (p.atomic) atomicAdd(dp + c, (Src)v);
                    else __stcs(dp + c, (Src)v);
                } else {
                    double v = 0;
                    if constexpr (kScale) {
                        if (c < po * (po + 1)) v = d_from_f_scaled(AR::ld(bp + c), eo * j + eo0);
                    } else if (c < po * (po + 1)) {
                        v = AR::to_d(AR::ld(bp + c));
                    }
                    if (c < pid * (pid + 1)) v += (double)__ldcs(sp + c);
                    if (p.atomic) atomicAdd(dp + c, (Src)v);
                    else __stcs(dp + c, (Src)((double)__ldcs(dp + c) + v));
                }
            }
        }
        __syncthreads();
    }
}

template <class A, int G, int ACC, bool FIX = false, bool HBM = true, bool WORK = false>
__global__ void __launch_bounds__(256) k_translate(KParams p)
{
    translate_body<A, G, ACC, FIX, HBM, WORK>(p);
}

// resident CTAs per SM that the registers have to allow
template <class A>
constexpr int fx_blocks(int acc)
{
    if (std::is_same<A, float>::value) return acc <= 4 ? 8 : acc <= 6 ? 6 : acc <= 8 ? 5 : acc <= 10 ? 4 : 2;
    return acc <= 4 ? 5 : acc <= 6 ? 4 : 2;
}
// FP64 in 60-bit block fixed point (A = double), FP32 (A = float)
template <class A, int G, int ACC, bool HBM = true, bool WORK = false>
__global__ void __launch_bounds__(kFxThreads, fx_blocks<A>(ACC)) k_translate_fx(KParams p)
{
    translate_body<A, G, ACC, true, HBM, WORK>(p);
}

// Resident CTAs per SM that the registers have to allow.  Four threads per
// translation: four CTAs at orders up to 4 (P=2 291 us, 327 with three), three
// at 5 to 8 (four spill 148 bytes: orders 2 to 6 in one launch 688 us, 621 with
// three, whose 16 bytes lie outside the stages), two at 9 to 16 (P=12 206 M/s,
// 166 with three).  Eight threads at orders 25 to 28: not more registers than
// twelve warps leave each other (168; with 179 only eight of the ten that shared
// memory allows were resident, P=25 1.83 ms, 1.55 so).
constexpr int split_blocks(int G, int acc)
{
    return G == 4 ? (acc <= 1 ? 4 : acc <= 2 ? 3 : acc <= 4 ? 2 : 1) : acc <= 2 ? 3 : acc == 3 ? 2 : 1;
}
constexpr int split_threads(int G, int acc) { return G == 8 && acc == 4 ? 384 : 256; }
// split precision
template <int G, int ACC, bool HBM = true, bool WORK = false>
__global__ void __launch_bounds__(split_threads(G, ACC), split_blocks(G, ACC)) k_translate_split(KParams p)
{
    translate_body<ff, G, ACC, true, HBM, WORK>(p);
}

}  // namespace sfmm
