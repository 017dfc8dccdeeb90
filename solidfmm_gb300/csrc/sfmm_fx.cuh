// Plain FP64 translations in 60-bit block fixed point.
//
// The swaps are orthogonal and the azimuthal and polar rotations unitary, so
// one degree of an expansion (a "row": its real and imaginary parts in the
// orthogonal basis) keeps its 2-norm from the forward edge to the last swap.
// A row therefore runs on int64 mantissas that share one block exponent,
// M = value / 2^E, entering with |M| <= 2^(60-hb), 2^hb >= sqrt(2 d): every
// intermediate then stays within 2^60 and no stage has to renormalise.  The
// constants (swap matrices, cos / sin, edge factors) are 60-bit fixed point.
// Mantissas and constants are split M = h 2^30 + l with l in [-2^29, 2^29),
// and a sum of products is
//     sum w x = sum wh xh + (sum (wh xl + wl xh) + 2^29 >> 30)
// in units of 2^E: three 32x32+64-bit multiply-adds per term, exact except
// for the wl xl terms (below 2^-2 d units) and one rounding of half a unit.
// Bounds: sum wh xh <= 2^60 (Cauchy-Schwarz, unit rows), and the cross sum is
// at most 2^60 sqrt(d/2) < 2^63 for every d <= 96.  One unit is 2^-57 (d <=
// 32) of the row's largest element, against 2^-53 for FP64's own roundings.
//
// On GB300 an FP64 multiply-add occupies its pipe for 64 cycles per warp and
// scheduler, an integer 32x32+64-bit one for four: three of them per term leave
// the FP64 pipe to the z-translation, whose coefficients span too many orders of
// magnitude for a block exponent, and to the accumulation into the targets.
// Measured (M2L, one GB300): P=16 37.1 -> 86.2 M/s, P=8 168 -> 387, P=24 11.7
// -> 22.1, with an error no larger than the FP64 transforms' (P=16 M2L 2.1e-15
// against 3.4e-15, M2M 7.1e-17 against 9.1e-17, P=21 L2L 2e-16 against 4.5e-15).
// What bounds it now: the FP64 pipe is busy 55% of
// the time with the z-translation alone, the schedulers issue in 45% of the
// cycles with 20 resident warps (registers and shared memory).
//
// Lane layout: lane q of a translation's G lanes holds part q & 1 (real or
// imaginary) of the rows m = (q >> 1) + (G/2) a, a < NA = ceil(d / (G/2)).
// The rotations mix the two parts of an element, which neighbouring lanes
// exchange by shuffles.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "sfmm_arith.cuh"
#include "sfmm_params.hpp"

namespace sfmm {

template <int N>
struct ic {
    static constexpr int value = N;
};

constexpr int kFxNone = -(1 << 20);  // exponent of no element
constexpr int kFxBad = 1 << 20;      // exponent of a non-finite element

// mantissa h 2^30 + l
struct fx {
    int h, l;
};

// A mantissa M is split from M + 2^29 (l centred, what a swap's cross sums
// need) or from M itself (l in [0, 2^30), enough for a product of two); the
// accumulations that produce M take the 2^29 into their initial value.
constexpr long long kFxRound = 1ll << 29;                        // of the cross sums
constexpr long long kFxRoundCentred = kFxRound + (1ll << 59);    // the same, adding 2^29 to the result
__device__ __forceinline__ fx fx_split_centred(long long m) { return fx{(int)(m >> 30), ((int)m & 0x3fffffff) - (1 << 29)}; }
__device__ __forceinline__ fx fx_split(long long m) { return fx{(int)(m >> 30), (int)m & 0x3fffffff}; }

// positive scalar (m / 2^60) 2^e with m in [2^59, 2^60]
struct fxs {
    fx m;
    int e;
};

// a b as one 32x32->64-bit product, which fuses with the addition around it
// (as C++, products of limbs just shifted out of a 64-bit word become
// 64x64-bit ones, and mad.wide in PTX keeps the addition apart)
__device__ __forceinline__ long long mul_wide(int a, int b)
{
    long long d;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) { return mul_wide(a, b) + c; }

// a b / 2^60, rounded
__device__ __forceinline__ long long fx_mul(fx a, fx b)
{
    const long long c = mad_wide(a.h, b.l, mad_wide(a.l, b.h, kFxRound));
    return mad_wide(a.h, b.h, c >> 30);
}

// (c x + s y) / 2^60, rounded (with round = kFxRoundCentred: plus 2^29)
__device__ __forceinline__ long long fx_dot2(fx c, fx x, fx s, fx y, long long round = kFxRound)
{
    const long long t = mad_wide(c.h, x.l, mad_wide(c.l, x.h, mad_wide(s.h, y.l, mad_wide(s.l, y.h, round))));
    return mad_wide(c.h, x.h, mad_wide(s.h, y.h, t >> 30));
}

__device__ __forceinline__ fx fx_neg(fx a) { return fx{-a.h, -a.l}; }
__device__ __forceinline__ fx fx_partner(fx a)
{
    return fx{__shfl_xor_sync(0xffffffffu, a.h, 1), __shfl_xor_sync(0xffffffffu, a.l, 1)};
}

__device__ __forceinline__ fxs fxs_mul(fxs a, fxs b)
{
    long long m = fx_mul(a.m, b.m);  // [2^58, 2^60]
    int e = a.e + b.e;
    if (m < (1ll << 59)) {
        m <<= 1;
        --e;
    }
    return fxs{fx_split(m), e};
}

// |x| = (m / 2^60) 2^(eb - 1022), m in [2^59, 2^60) for normal x, eb = max(1,
// the biased exponent field), 0x7ff for infinities and NaN
struct fxd {
    unsigned mh, ml;  // the 53-bit significand
    int eb;
    int neg;  // -1 or 0
};
__device__ __forceinline__ fxd fx_unpack(double x)
{
    const unsigned hw = (unsigned)__double2hiint(x);
    const int ef = (int)(hw >> 20 & 0x7ffu);
    return fxd{(hw & 0xfffffu) | (ef ? 0x100000u : 0u), (unsigned)__double2loint(x), max(ef, 1), (int)hw >> 31};
}
// its 60-bit mantissa, as limbs (l in [0, 2^30)) and as one word
__device__ __forceinline__ fx fx_limbs(fxd v) { return fx{(int)__funnelshift_l(v.ml, v.mh, 9), (int)(v.ml << 9 >> 2)}; }
__device__ __forceinline__ long long fx_word(fxd v)
{
    return (long long)((unsigned long long)__funnelshift_l(v.ml, v.mh, 7) << 32 | (v.ml << 7));
}

// int64 fixed-point coefficient of a double in [-1, 1]
__device__ __forceinline__ long long fx_q60(double x)
{
    const fxd v = fx_unpack(x);
    const int e = v.eb - 1022;
    const long long m = fx_word(v), r = e <= 0 ? m >> min(-e, 63) : m << 1;  // |x| = 1: e = 1
    return v.neg ? -r : r;
}

// M 2^E, |M| < 2^62, rounded to nearest (ties away), for E in [-1000, 950]
// (every result is zero or normal)
__device__ __forceinline__ double fx_to_double(long long M, int E)
{
    const int sg = (int)(M >> 32) >> 31;
    const unsigned long long a = (unsigned long long)((M ^ (long long)sg) - (long long)sg);
    const int lz = __clzll((long long)a) - 1;                 // >= 1; 63 for zero
    const unsigned long long r = ((a << lz) + 0x200u) >> 10;  // [2^52, 2^53]
    const unsigned hi = (unsigned)(r >> 32) + ((unsigned)(1023 + 61 - lz + E) << 20);  // hidden bit adds 1 to the exponent
    return M ? __hiloint2double((int)(hi | ((unsigned)sg & 0x80000000u)), (int)(unsigned)r) : 0.0;
}
__device__ __forceinline__ bool fx_safe(int E) { return (unsigned)(E + 800) < 1600u; }
// the same for any E (rows of tiny or huge coefficients)
__device__ __forceinline__ double fx_to_double_any(long long M, int E)
{
    E = max(-2400, min(2400, E));
    const int k = E / 4;
    const double f = __hiloint2double((1023 + k) << 20, 0);
    return fx_to_double(M, E - 3 * k) * f * f * f;
}

template <int G>
__device__ __forceinline__ int group_max_int(int v)
{
#pragma unroll
    for (int o = 1; o < G; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ void fx_store(double *p, fx v) { *reinterpret_cast<int2 *>(p) = make_int2(v.h, v.l); }

// cos and signed sin of m alpha and m beta for the rows of a lane, the sine
// signed so that own' = c own + s other is the rotation by +angle in either
// part (the backward rotations negate it)
template <int ACC>
struct FxTrig {
    fx ca[ACC], sa[ACC], cb[ACC], sb[ACC];
};

// (c, s) of unit length but for the roundings of two doubles, made one to a few
// units of 2^-60.  A translation rotates back what it rotated forth, so the
// error in length of (c, s) enters element m of its result m times over; the
// angle's own rounding mostly cancels.
__device__ __forceinline__ void fx_unit(long long &c, long long &s)
{
    const fx cl = fx_split_centred(c + (1 << 29)), sl = fx_split_centred(s + (1 << 29));
    const long long d = fx_dot2(cl, cl, sl, sl) - (1ll << 60);  // c^2 + s^2 - 1
    if (d > -(1 << 20) && d < (1 << 20)) {
        c -= mul_wide(cl.h, (int)d) >> 31;
        s -= mul_wide(sl.h, (int)d) >> 31;
    }
}

// Per-translation geometry, computed once per tile by one thread each.
// From the shift (already negated for M2M).  The components are scaled by a
// power of two first, so that squares neither overflow nor underflow; the
// transverse ones by their own, since (cos, sin) of the azimuth are as long as
// 1 only while no square underflows beside a far larger z.
__device__ __forceinline__ void fx_geometry(double x, double y, double z, FxGeo *out)
{
    const int ka = max(exp_of(x), exp_of(y)), k = max(ka, exp_of(z));
    const double xa = d_scaled(x, -ka), ya = d_scaled(y, -ka), zs = d_scaled(z, -k);
    const double ra2 = fma(xa, xa, ya * ya), ra = sqrt(ra2);
    const double rxy = d_scaled(ra, ka - k);
    const double r = sqrt(fma(zs, zs, d_scaled(ra2, 2 * (ka - k))));
    const double rinv = 1.0 / r;
    double ca = 1.0, sa = 0.0;
    if (ra > 0) {
        const double ri = 1.0 / ra;
        ca = ya * ri;
        sa = xa * ri;
    }
    FxGeo g;
    g.ca = fx_q60(ca);
    g.sa = fx_q60(sa);
    g.cb = fx_q60(zs * rinv);
    g.sb = fx_q60(-rxy * rinv);
    fx_unit(g.ca, g.sa);
    fx_unit(g.cb, g.sb);
    const fxd vr = fx_unpack(r), vi = fx_unpack(rinv);
    g.r = fx_word(vr);
    g.rinv = fx_word(vi);
    g.re = vr.eb - 1022 + k;
    g.rinve = vi.eb - 1022 - k;
    if (!(r > 0.0) || !isfinite(r)) g.re = g.rinve = kFxBad;
    else {
        // r / r = 1 to 2^-59 instead of 2^-53: M2M and L2L multiply by r^n and
        // r^-n.  r is in [1, 4), so the words' product is 1 / 2 or 1 / 4.
        const int e = vr.eb + vi.eb - 2044;
        const long long d = fx_mul(fx_split(g.r), fx_split(g.rinv)) - (1ll << (60 - e));
        g.rinv = max(g.rinv - (mul_wide((int)(g.rinv >> 30), (int)d) >> (30 - e)), 1ll << 59);
    }
    *out = g;
}

// e^{i m gamma} for m = r + RS a: binary powers for r, then steps of RS
template <int RS, int ACC>
__device__ __forceinline__ void fx_powers(long long c1, long long s1, int r, int part, fx (&c)[ACC], fx (&s)[ACC])
{
    fx kc = fx_split_centred(c1 + (1 << 29)), ks = fx_split_centred(s1 + (1 << 29));
    fx pc{1 << 30, 0}, ps{0, 0};
#pragma unroll
    for (int bit = 1; bit < RS; bit <<= 1) {
        if (r & bit) {
            const long long nc = fx_dot2(pc, kc, fx_neg(ps), ks, kFxRoundCentred), ns = fx_dot2(ps, kc, pc, ks, kFxRoundCentred);
            pc = fx_split_centred(nc);
            ps = fx_split_centred(ns);
        }
        const long long nc = fx_dot2(kc, kc, fx_neg(ks), ks, kFxRoundCentred), ns = fx_dot2(ks, kc, kc, ks, kFxRoundCentred);
        kc = fx_split_centred(nc);
        ks = fx_split_centred(ns);
    }
#pragma unroll
    for (int a = 0; a < ACC; ++a) {
        c[a] = pc;
        s[a] = part ? ps : fx_neg(ps);  // im' = c im + s re, re' = c re - s im
        if (a + 1 < ACC) {
            const long long nc = fx_dot2(pc, kc, fx_neg(ps), ks, kFxRoundCentred), ns = fx_dot2(ps, kc, pc, ks, kFxRoundCentred);
            pc = fx_split_centred(nc);
            ps = fx_split_centred(ns);
        }
    }
}

// One swap of a degree: rows m = r + RS a of W_R (part 0) or W_I (part 1)
// applied to the mantissas of the lane's part.  The coefficients of column
// slot t (column j0 + 2t, j0 = (r + n + part) & 1) lie together, lane by
// lane: NA/2 int4 per lane for pairs of rows, then an int2 for an odd last
// one, so a lane fetches two rows by one 16-byte load.
template <int G, int NA>
__device__ __forceinline__ void swap_fx(const int2 *__restrict__ W, const double *own, int j0, int cnt, int q,
                                        long long round, long long (&out)[NA])
{
    constexpr int NP = NA / 2;
    const int2 *x = reinterpret_cast<const int2 *>(own) + j0;
    const int4 *w4 = reinterpret_cast<const int4 *>(W) + q;
    const int2 *w2 = W + 2 * NP * G + q;
    long long A[NA], C[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        A[a] = 0;
        C[a] = round;
    }
#pragma unroll 2
    for (int t = 0; t < cnt; ++t) {
        const int2 v = *x;
        int2 w[NA];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int4 u = __ldg(w4 + p * G);
            w[2 * p] = make_int2(u.x, u.y);
            w[2 * p + 1] = make_int2(u.z, u.w);
        }
        if constexpr (NA & 1) w[NA - 1] = __ldg(w2);
        x += 2;
        w4 += NA * G / 2;
        w2 += NA * G;
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            A[a] += mul_wide(w[a].x, v.x);
            C[a] += mul_wide(w[a].x, v.y);
            C[a] += mul_wide(w[a].y, v.x);
        }
    }
#pragma unroll
    for (int a = 0; a < NA; ++a) out[a] = A[a] + (C[a] >> 30);
}

// row exponent (largest over the group) -> block exponent and shift base
__device__ __forceinline__ int fx_headroom(int d) { return d <= 2 ? 1 : d <= 8 ? 2 : d <= 32 ? 3 : 4; }

// one row: doubles from the mantissas M 2^E (NaN for a bad row); safe: every
// exponent is far from the ends of the FP64 range.  Zeros need no exponent:
// the rows above a source's own order take the fast form too.
template <int G, int NA>
__device__ __forceinline__ void fx_store_row(double *own, int d, int r, const long long (&M)[NA], const int (&E)[NA],
                                             bool safe, bool bad)
{
    constexpr int RS = G / 2;
    if (!safe) {
        long long any = 0;
#pragma unroll
        for (int a = 0; a < NA; ++a) any |= M[a];
        safe = any == 0;
    }
    if (safe && !bad) {
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const double v = fx_to_double(M[a], E[a]);
            if (a + 1 < NA || r + RS * a < d) own[r + RS * a] = v;
        }
    } else {
#pragma unroll 1
        for (int a = 0; a < NA; ++a) {
            long long v = M[0];
            int e = E[0];
#pragma unroll
            for (int i = 1; i < NA; ++i) {
                v = a == i ? M[i] : v;
                e = a == i ? E[i] : e;
            }
            if (r + RS * a < d) own[r + RS * a] = bad ? __hiloint2double(0x7ff80000, 0) : fx_to_double_any(v, e);
        }
    }
}

// Rows next to the smallest doubles.  Subnormals have fewer bits than their
// exponent says, and an edge factor (2^-142 to 2^142) may raise them to any
// size; a zero counts with the exponent 1 and its edge factor's.  Neither
// reaches the block exponent of a row whose largest element has a biased
// exponent above kFxTiny.  The gather looks for coefficients up to there, and
// takes rows that have no larger one times 2^kFxRaise.
constexpr int kFxTiny = 406;
constexpr int kFxRaise = 600;
// The running minimum over coefficients that finds them: the high word less
// one, zeros above all others.
__device__ __forceinline__ unsigned fx_low(double x, unsigned low)
{
    return min(low, (((unsigned)__double2hiint(x) & 0x7fffffffu) | min((unsigned)__double2loint(x), 1u)) - 1u);
}
__device__ __forceinline__ bool fx_tiny(unsigned low) { return low < (unsigned)(kFxTiny + 1) << 20; }
// The degrees raised are noted in the last word of the buffer's padding, which
// the swaps multiply by zero coefficients only.
__device__ __forceinline__ int fx_raised(const double *b, int spad, int n)
{
    return *reinterpret_cast<const unsigned *>(b + spad - 1) >> n & 1u ? kFxRaise : 0;
}
// One expansion of order P by one warp.
__device__ __forceinline__ void fx_raise_rows(double *b, int spad, int P, int lane)
{
    unsigned raised = 0;
    __syncwarp();
#pragma unroll 1
    for (int n = 0; n < P; ++n) {
        const int d = n + 1;
        double *row = b + n * d;
        int top = kFxNone;
        for (int c = lane; c < 2 * d; c += 32) {
            const fxd x = fx_unpack(c == d ? 0.0 : row[c]);  // the imaginary part at m = 0 is zero
            if (x.mh | x.ml) top = max(top, x.eb);
        }
        top = group_max_int<32>(top);
        if (top == kFxNone || top > kFxTiny) continue;
        for (int c = lane; c < 2 * d; c += 32) row[c] *= __hiloint2double((1023 + kFxRaise) << 20, 0);
        raised |= 1u << n;
    }
    if (lane == 0) *reinterpret_cast<unsigned *>(b + spad - 1) = raised;
}

// One degree of the forward transform: edge (r-power and basis factor g, one
// product per element), rotation by alpha, swap, rotation by beta, swap;
// doubles in, doubles out.
template <int G, int NA, int ACC>
__device__ __forceinline__ void forward_degree_fx(double *b, int n, const int2 *__restrict__ W,
                                                  const int4 *__restrict__ ein, fxs f, bool bad, int spad,
                                                  int q, const FxTrig<ACC> &tg)
{
    constexpr int RS = G / 2;
    const int d = n + 1, r = q >> 1, part = q & 1, j0 = (r + n + part) & 1, cnt = (d + 1) >> 1;
    double *own = b + n * d + part * d;
    long long p[NA];
    int e[NA];
    int emax = kFxNone;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const bool on = (a + 1 < NA || m < d) && (a || m || !part);  // the imaginary part at m = 0 is zero
        const fxd x = fx_unpack(on ? own[m] : 0.0);
        const int4 t = __ldg(ein + (a + 1 < NA ? m : min(m, n)));
        fx g = fx_split(fx_mul(f.m, fx{t.x, t.y}));
        g.h = (g.h ^ x.neg) - x.neg;
        g.l = (g.l ^ x.neg) - x.neg;
        p[a] = fx_mul(fx_limbs(x), g);
        e[a] = x.eb + t.z;
        bad |= x.eb == 0x7ff;
        emax = max(emax, e[a]);
    }
    emax = group_max_int<G>(bad ? kFxBad : emax);
    bad = emax == kFxBad;
    const int hb = fx_headroom(d);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const fx v = fx_split(p[a] >> min(emax - e[a] + hb, 63));
        const fx o = fx_partner(v);
        if (a + 1 < NA || m < d) fx_store(own + m, fx_split_centred(fx_dot2(tg.ca[a], v, tg.sa[a], o, kFxRoundCentred)));
    }
    __syncwarp();
    long long M[NA];
    swap_fx<G, NA>(W, own, j0, cnt, q, kFxRound, M);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const fx v = fx_split(M[a]);
        const fx o = fx_partner(v);
        if (a + 1 < NA || m < d) fx_store(own + m, fx_split_centred(fx_dot2(tg.cb[a], v, tg.sb[a], o, kFxRoundCentred)));
    }
    __syncwarp();
    swap_fx<G, NA>(W, own, j0, cnt, q, kFxRound, M);
    __syncwarp();
    const int E = emax + f.e - 1022 - 60 + hb - fx_raised(b, spad, n);
    int Ea[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) Ea[a] = E;
    fx_store_row<G, NA>(own, d, r, M, Ea, fx_safe(E), bad);
    __syncwarp();
}

// One degree of the backward transform: swap, rotation by -beta, swap,
// rotation by -alpha, edge.
template <int G, int NA, int ACC>
__device__ __forceinline__ void backward_degree_fx(double *b, int n, const int2 *__restrict__ W,
                                                   const int4 *__restrict__ eout, fxs f, bool bad, int q,
                                                   const FxTrig<ACC> &tg)
{
    constexpr int RS = G / 2;
    const int d = n + 1, r = q >> 1, part = q & 1, j0 = (r + n + part) & 1, cnt = (d + 1) >> 1;
    double *own = b + n * d + part * d;
    long long p[NA];
    int e[NA];
    int emax = kFxNone;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const fxd x = fx_unpack(a + 1 < NA || m < d ? own[m] : 0.0);
        p[a] = (fx_word(x) ^ (long long)x.neg) - (long long)x.neg;
        e[a] = x.eb;
        emax = max(emax, e[a]);
    }
    emax = group_max_int<G>(bad ? kFxBad : emax);
    bad = emax >= 0x7ff;
    const int hb = fx_headroom(d);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        if (a + 1 < NA || m < d) fx_store(own + m, fx_split_centred((p[a] >> min(emax - e[a] + hb, 63)) + (1ll << 29)));
    }
    __syncwarp();
    long long M[NA];
    swap_fx<G, NA>(W, own, j0, cnt, q, kFxRound, M);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const fx v = fx_split(M[a]);
        const fx o = fx_neg(fx_partner(v));
        if (a + 1 < NA || m < d) fx_store(own + m, fx_split_centred(fx_dot2(tg.cb[a], v, tg.sb[a], o, kFxRoundCentred)));
    }
    __syncwarp();
    swap_fx<G, NA>(W, own, j0, cnt, q, kFxRound, M);
    __syncwarp();
    const int E = emax + f.e - 1022 - 60 + hb;
    int Ea[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = r + RS * a;
        const fx v = fx_split(M[a]);
        const fx o = fx_neg(fx_partner(v));
        const int4 t = __ldg(eout + (a + 1 < NA ? m : min(m, n)));
        const fx g = fx_split(fx_mul(f.m, fx{t.x, t.y}));
        M[a] = fx_mul(fx_split(fx_dot2(tg.ca[a], v, tg.sa[a], o)), g);
        Ea[a] = E + t.z;
    }
    fx_store_row<G, NA>(own, d, r, M, Ea, fx_safe(E), bad);
    __syncwarp();
}

// V = 16 / sizeof(T) consecutive row blocks of a z matrix row come by one load
template <class T>
constexpr int kZVec = 16 / (int)sizeof(T);
template <class T>
struct zvec;
template <>
struct zvec<double> {
    using type = double2;
    static __device__ __forceinline__ void get(const type &v, double *w)
    {
        w[0] = v.x;
        w[1] = v.y;
    }
};
template <>
struct zvec<float> {
    using type = float4;
    static __device__ __forceinline__ void get(const type &v, float *w)
    {
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
    }
};
// blocks [B0, B1) of one row into w[B0 ..] (w has room for whole vectors)
template <class T, int RS, int B0, int B1, int N>
__device__ __forceinline__ void z_load(const T *h, T (&w)[N])
{
    constexpr int V = kZVec<T>;
#pragma unroll
    for (int i = B0 / V; i < (B1 + V - 1) / V; ++i) {
        if (B1 - i * V == 1) w[i * V] = __ldg(h + i * RS * V);
        else zvec<T>::get(__ldg(reinterpret_cast<const typename zvec<T>::type *>(h + i * RS * V)), w + i * V);
    }
}

// One z-translation column m: outputs n' = m + r + RS b (b < NB) of the
// lane's part, in(k, m) read once per row for all of them.  H_m lies row by
// row (k), in each row vectors of V blocks lane by lane, hs elements per row.
template <class T, int G, int NB>
__device__ __forceinline__ void z_column_part(T *b, const T *__restrict__ Hm, int hs, int m, int kend, int nout, int q)
{
    constexpr int RS = G / 2, V = kZVec<T>, NW = (NB + V - 1) / V * V;
    const int r = q >> 1, part = q & 1;
    T acc[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) acc[i] = 0;
    const T *h = Hm + V * r;
    int o = m * (m + 1) + m + part * (m + 1);
    int step = 2 * (m + 1) + part;
    T wn[NW], xn = b[o];
    z_load<T, RS, 0, NB>(h, wn);
#pragma unroll 2
    for (int k = m; k < kend; ++k) {  // row k+1's operands load before row k's multiply-adds
        const T x = xn;
        T w[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) w[i] = wn[i];
        if (k + 1 < kend) {
            o += step;
            step += 2;
            h += hs;
        }
        xn = b[o];
        z_load<T, RS, 0, NB>(h, wn);
#pragma unroll
        for (int i = 0; i < NB; ++i) acc[i] = fma(w[i], x, acc[i]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int np = m + r + RS * i;
        if (np < nout) b[np * (np + 1) + m + part * (np + 1)] = acc[i];
    }
    __syncwarp();
}

// The same for the triangular operators, with the products of the zero half
// left out: L2L needs rows k >= n', M2M rows k <= n'.  A lane walks its own
// rows, k = m + r + j upwards (L2L) or k = m + r + RS (NB - 1) - j downwards
// (M2M), so that with every RS rows one more block of outputs joins, for all
// lanes at once: 40 of 64 multiply-adds of a column of 16 remain.
template <class T, int G, int NB, bool UP>
__device__ __forceinline__ void z_column_tri(T *b, const T *__restrict__ Hm, int hs, int m, int kend, int nout, int q)
{
    constexpr int RS = G / 2, D = UP ? 1 : -1, V = kZVec<T>, NW = (NB + V - 1) / V * V;
    const int r = q >> 1, part = q & 1;
    T acc[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) acc[i] = 0;
    // rows that no lane has: above kend on the way down
    int j = UP ? 0 : max(0, m + RS * (NB - 1) - kend + 1);
    const int rows = UP ? kend - m : RS * NB;
    int k = m + r + (UP ? 0 : RS * (NB - 1) - j);
    const T *h = Hm + (long long)(k - m) * hs + V * r;
    int o = k * (k + 1) + m + part * (k + 1);
    int step = UP ? 2 * (k + 1) + part : 2 * k + part;  // to the next row (UP) or the previous one
    auto stage = [&](auto nb) {
        constexpr int N = decltype(nb)::value, B0 = UP ? 0 : NB - N, B1 = UP ? N : NB;  // blocks at work
        const int end = N < NB ? min(RS * N, rows) : rows;
#pragma unroll 2
        for (; j < end; ++j) {
            if (UP ? k < kend : k < kend && k >= m) {
                const T x = b[o];
                T w[NW];
                z_load<T, RS, B0, B1>(h, w);
#pragma unroll
                for (int i = B0; i < B1; ++i) acc[i] = fma(w[i], x, acc[i]);
            }
            k += D;
            o += D * step;
            step += 2 * D;
            h += D * hs;
        }
    };
    stage(ic<1>{});
    if constexpr (NB >= 2) stage(ic<2>{});
    if constexpr (NB >= 3) stage(ic<3>{});
    if constexpr (NB >= 4) stage(ic<4>{});
    if constexpr (NB >= 5) stage(ic<5>{});
    if constexpr (NB >= 6) stage(ic<6>{});
    if constexpr (NB >= 7) stage(ic<7>{});
    if constexpr (NB >= 8) stage(ic<8>{});
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int np = m + r + RS * i;
        if (np < nout) b[np * (np + 1) + m + part * (np + 1)] = acc[i];
    }
    __syncwarp();
}

// Column m of operator op.
template <class T, int G, int NB>
__device__ __forceinline__ void z_column_op(int op, T *b, const T *__restrict__ Hm, int hs, int m, int pin, int pout, int q)
{
    if (op == OP_M2L) z_column_part<T, G, NB>(b, Hm, hs, m, pin, pout, q);
    else if (op == OP_L2L) z_column_tri<T, G, NB, true>(b, Hm, hs, m, pin, pout, q);
    else z_column_tri<T, G, NB, false>(b, Hm, hs, m, min(pin, pout), pout, q);
}

}  // namespace sfmm
