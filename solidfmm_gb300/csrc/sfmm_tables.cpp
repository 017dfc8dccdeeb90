#include "sfmm_tables.hpp"

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "sfmm_fx_layout.hpp"

namespace sfmm {

std::vector<std::vector<double>> swap_matrices(int P)
{
    std::vector<std::vector<double>> B(P > 0 ? P : 0);
    auto b = [&](int n, int m, int l) -> double {
        if (n < 0 || std::abs(l) > n || std::abs(m) > n) return 0.0;
        return B[n][(m + n) + (l + n) * (2 * n + 1)];
    };
    for (int n = 0; n < P; ++n) {
        int w = 2 * n + 1;
        B[n].assign(size_t(w) * w, 0.0);
        auto at = [&](int m, int l) -> double & { return B[n][(m + n) + (l + n) * w]; };
        if (n == 0) {
            at(0, 0) = 1;
            continue;
        }
        // recursion in the degree (swap_matrix.cpp:155-170)
        for (int l = -n; l <= n; ++l) at(0, l) = 0.5 * (b(n - 1, 0, l - 1) - b(n - 1, 0, l + 1));
        for (int m = 0; m < n; ++m)
            for (int l = -n; l <= n; ++l) {
                at(m + 1, l) = 0.5 * (b(n - 1, m, l - 1) + b(n - 1, m, l + 1)) + b(n - 1, m, l);
                at(-m - 1, l) = 0.5 * (b(n - 1, -m, l - 1) + b(n - 1, -m, l + 1)) - b(n - 1, -m, l);
            }
    }
    return B;
}

namespace {

// sqrt(k!) in FP64 (k! itself is finite up to 170!, the largest the
// tables need for P <= 86).
struct SqrtFac {
    std::vector<double> v;
    explicit SqrtFac(int kmax) : v(kmax + 1)
    {
        double f = 1;
        for (int k = 0; k <= kmax; ++k) {
            if (k) f *= k;
            v[k] = std::sqrt(f);
        }
    }
    double operator()(int k) const { return v[k]; }
};

}  // namespace

double w_entry(const HostTables &t, int n, int part, int i, int j)
{
    const int d = n + 1, R = wrows(d, t.pad);
    if (i < 0 || j < 0 || i >= d || j >= d) return 0.0;
    const bool rnz = ((i + j + n) & 1) == 0;
    if (rnz != (part == 0)) return 0.0;
    return t.W[t.woff[n] + size_t(j >> 1) * 2 * R + (part ? R : 0) + i];
}

namespace {

// Swap blocks of degrees n < nmax with rows padded to a multiple of pad (the
// layout of HostTables::W).
void build_w(const std::vector<std::vector<double>> &B, const SqrtFac &sf, int nmax, int pad,
             std::vector<double> &W, std::vector<int> &woff)
{
    const double s2 = std::sqrt(2.0);
    woff.resize(nmax);
    size_t tot = 0;
    for (int n = 0; n < nmax; ++n) {
        woff[n] = (int)tot;
        tot += 2 * size_t(wcols(n + 1)) * wrows(n + 1, pad);
    }
    W.assign(tot, 0.0);
    for (int n = 0; n < nmax; ++n) {
        const int d = n + 1, w = 2 * n + 1;
        auto Bv = [&](int m, int l) { return B[n][(m + n) + (l + n) * w]; };
        auto D = [&](int m) { return sf(n - m) * sf(n + m); };
        auto E = [&](int m) { return m == 0 ? D(0) / s2 : D(m); };
        const int R = wrows(d, pad);
        double *WR = &W[woff[n]];  // slot t: W_R rows at 2tR, W_I rows at 2tR + R
        double *WI = WR + R;
        for (int i = 0; i < d; ++i)       // output row (coefficient m = i)
            for (int j = 0; j < d; ++j) { // input column (coefficient l = j)
                // the reference's real/imag combinations (operator_data.cpp:99-147)
                double rf, imf;
                if (j == 0) rf = Bv(0, i);
                else if (j & 1) rf = Bv(j, i) - Bv(-j, i);
                else rf = Bv(j, i) + Bv(-j, i);
                if (j & 1) imf = Bv(j, i) + Bv(-j, i);
                else imf = Bv(j, i) - Bv(-j, i);
                // keep only the checkerboard the reference stores
                const bool rnz = ((i + j + n) & 1) == 0;
                const size_t slot = size_t(j >> 1) * 2 * R + i;  // j = jr(i) + 2t or ji(i) + 2t
                if (rnz) WR[slot] = rf * (E(i) / E(j));
                else if (i > 0 && j > 0) WI[slot] = imf * (D(i) / D(j));
            }
    }
}

}  // namespace

HostTables build_tables(int P)
{
    HostTables t;
    t.P = P;
    const int pad = row_pad(P);
    t.pad = pad;
    auto B = swap_matrices(P);
    SqrtFac sf(2 * P + 2);
    std::vector<double> fac(2 * P + 2);
    fac[0] = 1;
    for (int k = 1; k < 2 * P + 2; ++k) fac[k] = fac[k - 1] * k;
    const double s2 = std::sqrt(2.0);

    build_w(B, sf, P, pad, t.W, t.woff);
    if (pad != 8) build_w(B, sf, std::min(P, 32), 8, t.W8, t.woff8);

    size_t ne = size_t(P) * (P + 1) / 2;
    t.e_in_M.resize(ne);
    t.e_in_L.resize(ne);
    t.e_out_L.resize(ne);
    t.e_out_M.resize(ne);
    for (int n = 0; n < P; ++n)
        for (int m = 0; m <= n; ++m) {
            double D = sf(n - m) * sf(n + m);
            double s = m == 0 ? s2 : 1.0;
            size_t k = size_t(n) * (n + 1) / 2 + m;
            t.e_in_M[k] = D / s;
            t.e_in_L[k] = 1.0 / (D * s);
            t.e_out_L[k] = D * s;
            t.e_out_M[k] = s / D;
        }

    t.hoff.resize(P);
    size_t th = 0;
    for (int m = 0; m < P; ++m) {
        t.hoff[m] = (int)th;
        th += size_t(P - m + 2) * hrows(P - m, pad);
    }
    for (int op = 0; op < 3; ++op) t.H[op].assign(th, 0.0);
    for (int m = 0; m < P; ++m) {
        const int HR = hrows(P - m, pad);
        for (int k = m; k < P; ++k)
            for (int np = m; np < P; ++np) {
                size_t idx = t.hoff[m] + size_t(k - m) * HR + (np - m);
                double Dk = sf(k - m) * sf(k + m);
                double Dn = sf(np - m) * sf(np + m);
                // M2L: (-1)^(n'+m) (n'+k)! / (D^(n') D^(k))   (zm2l, translations.cpp:283-296)
                double h1 = fac[np + k] / Dn / Dk;
                t.H[1][idx] = ((np + m) & 1) ? -h1 : h1;
                // M2M: D^(n') / ((n'-k)! D^(k)), k <= n'   (zm2m, translations.cpp:366-377)
                if (k <= np) t.H[0][idx] = Dn / (fac[np - k] * Dk);
                // L2L: D^(k) / (D^(n') (k-n')!), k >= n'   (zm2m, translations.cpp:440-451)
                if (k >= np) t.H[2][idx] = Dk / (Dn * fac[k - np]);
            }
    }
    return t;
}

namespace {

void put_fx(int32_t *at, double v, int scale)
{
    const int64_t m = std::llround(std::ldexp(v, scale));
    const int64_t h = (m + (int64_t(1) << 29)) >> 30;
    at[0] = (int32_t)h;
    at[1] = (int32_t)(m - h * (int64_t(1) << 30));
}

}  // namespace

FxTables build_fx_tables(const HostTables &t, int G, int P)
{
    FxTables f;
    f.P = P;
    const int RS = G / 2;
    f.woff.resize(P);
    size_t tot = 0;
    for (int n = 0; n < P; ++n) {
        f.woff[n] = (int)tot;
        tot += size_t((n + 2) / 2) * ((n + RS) / RS) * G;
    }
    f.W.assign(2 * tot, 0);
    for (int n = 0; n < P; ++n) {
        const int d = n + 1, NA = (d + RS - 1) / RS, cnt = (d + 1) / 2;
        for (int tt = 0; tt < cnt; ++tt)
            for (int q = 0; q < G; ++q)
                for (int a = 0; a < NA; ++a) {
                    const int part = q & 1, i = (q >> 1) + RS * a, j = ((i + n + part) & 1) + 2 * tt;
                    const size_t in_slot = a / 2 * 2 + 1 < NA ? size_t(a / 2 * G + q) * 2 + (a & 1) : size_t(NA - 1) * G + q;
                    put_fx(&f.W[2 * (f.woff[n] + size_t(tt) * NA * G + in_slot)], w_entry(t, n, part, i, j), 60);
                }
    }
    f.hoff.resize(P);
    tot = 0;
    for (int m = 0; m < P; ++m) {
        f.hoff[m] = (int)tot;
        tot += size_t(P - m) * fx_hrow(P - m, G);
    }
    for (int op = 0; op < 3; ++op) {
        f.H[op].assign(tot, 0.0);
        for (int m = 0; m < P; ++m) {
            const int HR = hrows(t.P - m, t.pad), hs = fx_hrow(P - m, G);
            for (int k = 0; k < P - m; ++k)
                for (int np = 0; np < P - m; ++np) {
                    const int r = np % RS, b = np / RS;
                    f.H[op][f.hoff[m] + size_t(k) * hs + b / 2 * G + 2 * r + (b & 1)] =
                        t.H[op][t.hoff[m] + size_t(k) * HR + np];
                }
        }
    }
    return f;
}

F32Tables build_f32_tables(const HostTables &t, int G, int P)
{
    F32Tables f;
    const int RS = G / 2;
    f.woff.resize(P);
    size_t tot = 0;
    for (int n = 0; n < P; ++n) {
        f.woff[n] = (int)tot;
        tot += size_t((n + 2) / 2) * (((n + RS) / RS + 3) / 4) * 4 * G;
    }
    f.W.assign(tot, 0.f);
    for (int n = 0; n < P; ++n) {
        const int d = n + 1, NA = (d + RS - 1) / RS, slot = (NA + 3) / 4 * 4 * G;
        for (int tt = 0; tt < (d + 1) / 2; ++tt)
            for (int q = 0; q < G; ++q)
                for (int a = 0; a < NA; ++a) {
                    const int part = q & 1, i = (q >> 1) + RS * a, j = ((i + n + part) & 1) + 2 * tt;
                    f.W[f.woff[n] + size_t(tt) * slot + a / 4 * 4 * G + 4 * q + a % 4] = (float)w_entry(t, n, part, i, j);
                }
    }
    f.hoff.resize(P);
    tot = 0;
    for (int m = 0; m < P; ++m) {
        f.hoff[m] = (int)tot;
        tot += size_t(P - m) * fx_hrow(P - m, G, 4);
    }
    for (int op = 0; op < 3; ++op) {
        f.H[op].assign(tot, 0.f);
        for (int m = 0; m < P; ++m) {
            const int HR = hrows(t.P - m, t.pad), hs = fx_hrow(P - m, G, 4);
            for (int k = 0; k < P - m; ++k)
                for (int np = 0; np < P - m; ++np) {
                    const int r = np % RS, b = np / RS;
                    f.H[op][f.hoff[m] + size_t(k) * hs + b / 4 * 2 * G + 4 * r + b % 4] =
                        (float)t.H[op][t.hoff[m] + size_t(k) * HR + np];
                }
        }
    }
    return f;
}

SplitTables build_split_tables(const HostTables &t, int G, int P)
{
    SplitTables f;
    f.woff.resize(P);
    size_t tot = 0;
    for (int n = 0; n < P; ++n) {
        f.woff[n] = (int)tot;
        tot += size_t((n + 2) / 2) * ((n + G) / G) * G;
    }
    f.W.assign(2 * (tot + size_t((P + G - 1) / G) * G), 0);  // and a slot that the last degree's loop loads ahead
    for (int n = 0; n < P; ++n) {
        const int d = n + 1, NA = (d + G - 1) / G;
        for (int tt = 0; tt < (d + 1) / 2; ++tt)
            for (int q = 0; q < G; ++q)
                for (int a = 0; a < NA; ++a) {
                    const int jr = (q + n) & 1, i = q + G * a;
                    const size_t in_slot = a / 2 * 2 + 1 < NA ? size_t(a / 2 * G + q) * 2 + (a & 1) : size_t(NA - 1) * G + q;
                    int32_t *at = &f.W[2 * (f.woff[n] + size_t(tt) * NA * G + in_slot)];
                    at[0] = (int32_t)std::llround(std::ldexp(w_entry(t, n, 0, i, jr + 2 * tt), 30));
                    at[1] = (int32_t)std::llround(std::ldexp(w_entry(t, n, 1, i, (jr ^ 1) + 2 * tt), 30));
                }
    }
    f.hoff.resize(P);
    tot = 0;
    for (int m = 0; m < P; ++m) {
        f.hoff[m] = (int)tot;
        tot += size_t(P - m) * fx_hrow(P - m, 2 * G);
    }
    for (int op = 0; op < 3; ++op) {
        f.H[op].assign(2 * tot, 0.f);
        for (int m = 0; m < P; ++m) {
            const int HR = hrows(t.P - m, t.pad), hs = fx_hrow(P - m, 2 * G);
            for (int k = 0; k < P - m; ++k)
                for (int np = 0; np < P - m; ++np) {
                    const int q = np % G, b = np / G;
                    const double v = t.H[op][t.hoff[m] + size_t(k) * HR + np];
                    float *at = &f.H[op][2 * (f.hoff[m] + size_t(k) * hs + b / 2 * 2 * G + 2 * q + (b & 1))];
                    at[0] = (float)v;
                    at[1] = (float)(v - (double)at[0]);
                }
        }
    }
    return f;
}

std::vector<int32_t> fx_edges(const std::vector<double> &e, size_t count)
{
    std::vector<int32_t> out(4 * count);
    for (size_t i = 0; i < count; ++i) {
        int ex;
        const double f = std::frexp(e[i], &ex);  // [1/2, 1)
        put_fx(&out[4 * i], f, 60);
        out[4 * i + 2] = ex;
    }
    return out;
}

}  // namespace sfmm
