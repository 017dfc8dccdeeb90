// Tables of the 60-bit fixed-point kernel (build_fx_tables, fx_edges) on the
// host: every swap coefficient, z-translation entry and edge factor is found
// where the kernel's lanes read it, equal to the context's FP64 tables (swap
// coefficients and edges to their rounding), rows and columns past a degree
// are zero, limbs are in range, and no offset leaves its table.  Prints "ok"
// and exits 0 on success.
#include <cmath>
#include <cstdio>
#include <vector>

#include "sfmm_fx_layout.hpp"
#include "sfmm_tables.hpp"

using namespace sfmm;

static int failures = 0;
#define CHECK(c, ...)                                   \
    do {                                                \
        if (!(c) && ++failures < 20) {                  \
            std::printf("FAIL %s: ", #c);               \
            std::printf(__VA_ARGS__);                   \
            std::printf("\n");                          \
        }                                               \
    } while (0)

static double value(const int32_t *p, int scale)
{
    return std::ldexp((double)p[0], 30 - scale) + std::ldexp((double)p[1], -scale);
}

int main()
{
    for (int P : {1, 3, 4, 13, 32, 40})
        for (int G : {4, 8}) {
            const HostTables t = build_tables(P);
            const int Q = P < 32 ? P : 32, RS = G / 2;
            const FxTables f = build_fx_tables(t, G, Q);
            for (int n = 0; n < Q; ++n) {
                const int d = n + 1, NA = (d + RS - 1) / RS, cnt = (d + 1) / 2;
                CHECK(2 * (f.woff[n] + (size_t)cnt * NA * G) == (n + 1 < Q ? 2 * (size_t)f.woff[n + 1] : f.W.size()),
                      "P=%d G=%d n=%d block end", P, G, n);
                CHECK(f.woff[n] % 2 == 0, "P=%d G=%d n=%d alignment of the 16-byte loads", P, G, n);
                for (int tt = 0; tt < cnt; ++tt)
                    for (int q = 0; q < G; ++q)
                        for (int a = 0; a < NA; ++a) {
                            const int part = q & 1, i = (q >> 1) + RS * a, j = (((q >> 1) + n + part) & 1) + 2 * tt;
                            // pairs of rows by one int4 per lane, an odd last row by an int2
                            const size_t base = f.woff[n] + (size_t)tt * NA * G;
                            const size_t at = a / 2 < NA / 2 ? base + ((size_t)(a / 2) * G + q) * 2 + a % 2
                                                             : base + (size_t)(NA / 2) * 2 * G + q;
                            const int32_t *c = &f.W[2 * at];
                            const double want = i < d && j < d ? w_entry(t, n, part, i, j) : 0.0;
                            CHECK(std::fabs(value(c, 60) - want) <= 0x1p-54, "P=%d G=%d n=%d (%d,%d)", P, G, n, i, j);
                            CHECK(c[0] >= -(1 << 30) && c[0] <= (1 << 30) && c[1] >= -(1 << 29) && c[1] <= (1 << 29),
                                  "P=%d G=%d n=%d (%d,%d) limbs", P, G, n, i, j);
                        }
            }
            for (int m = 0; m < Q; ++m) {
                const int hs = fx_hrow(Q - m, G);
                CHECK(f.hoff[m] % 2 == 0 && hs % 2 == 0, "P=%d G=%d m=%d alignment", P, G, m);
                CHECK(f.hoff[m] + (size_t)(Q - m) * hs <= f.H[0].size(), "P=%d G=%d m=%d end", P, G, m);
                CHECK(hs >= Q - m, "P=%d G=%d m=%d row", P, G, m);
                for (int op = 0; op < 3; ++op)
                    for (int k = m; k < Q; ++k)
                        for (int np = m; np < Q; ++np) {
                            const int r = (np - m) % RS, b = (np - m) / RS;
                            const double got = f.H[op][f.hoff[m] + (size_t)(k - m) * hs + b / 2 * G + 2 * r + b % 2];
                            const double want = t.H[op][t.hoff[m] + (size_t)(k - m) * hrows(P - m, t.pad) + (np - m)];
                            CHECK(got == want, "P=%d G=%d op=%d m=%d k=%d n'=%d", P, G, op, m, k, np);
                        }
            }
            for (const auto *e : {&t.e_in_M, &t.e_in_L, &t.e_out_L, &t.e_out_M}) {
                const size_t cnt = (size_t)Q * (Q + 1) / 2;
                const auto v = fx_edges(*e, cnt);
                CHECK(v.size() == 4 * cnt, "P=%d", P);
                for (size_t i = 0; i < cnt; ++i) {
                    CHECK(std::ldexp(value(&v[4 * i], 60), v[4 * i + 2]) == (*e)[i], "P=%d edge %zu", P, i);
                    CHECK(v[4 * i] >= (1 << 29) && v[4 * i] <= (1 << 30), "P=%d edge %zu normalised", P, i);
                }
            }
        }
    if (failures) return 1;
    std::printf("ok\n");
    return 0;
}
