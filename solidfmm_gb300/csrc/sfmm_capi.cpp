// C ABI of solidfmm-gb300 (include/sfmm.h): contexts, table upload, launch
// shapes and tuning, device-resident batches, P2M/P2L and evaluation entry
// points; batches in host memory are in sfmm_host.cpp.  No exception crosses
// this boundary.
#include "sfmm.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "sfmm_context.hpp"
#include "sfmm_launch.hpp"
#include "sfmm_params.hpp"
#include "sfmm_tables.hpp"

using namespace sfmm;

namespace sfmm {

int fail(sfmm_context *c, int st, const char *fmt, ...)
{
    if (c) {
        char b[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(b, sizeof b, fmt, ap);
        va_end(ap);
        c->err = b;
    }
    return st;
}

int cuda_fail(sfmm_context *c, cudaError_t e, const char *what)
{
    return fail(c, SFMM_CUDA_ERROR, "%s: %s", what, cudaGetErrorString(e));
}

size_t esize(Arith a) { return a == Arith::F32 ? sizeof(float) : (a == Arith::F64 ? sizeof(double) : 2 * sizeof(float)); }

namespace {

template <class T>
cudaError_t put(void **dst, const std::vector<T> &v)
{
    cudaError_t e = cudaMalloc(dst, v.empty() ? 16 : v.size() * sizeof(T));
    if (e == cudaSuccess && !v.empty()) e = cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
    return e;
}

}  // namespace

void free_arith(ArithTables &t)
{
    if (t.mem) cudaFree(t.mem);
    t = ArithTables{};
}

void free_tables(DevTables &t)
{
    void *ps[] = {t.W, t.ein_M, t.ein_L, t.eout_L, t.eout_M, t.H[0], t.H[1], t.H[2]};
    for (void *p : ps)
        if (p) cudaFree(p);
    t = DevTables{};
}

namespace {

void free_offsets(sfmm_context *c)
{
    for (int **p : {&c->d_woff, &c->d_hoff}) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
}

}  // namespace

namespace {

// tables of FP64 above order 32
int ensure_high(sfmm_context *c)
{
    DevTables &t = c->tab;
    if (t.ready) return SFMM_OK;
    cudaError_t e = put((void **)&c->d_woff, c->host.woff);
    if (e == cudaSuccess) e = put((void **)&c->d_hoff, c->host.hoff);
    if (e == cudaSuccess) e = put(&t.W, c->host.W);
    if (e == cudaSuccess) e = put(&t.ein_M, c->host.e_in_M);
    if (e == cudaSuccess) e = put(&t.ein_L, c->host.e_in_L);
    if (e == cudaSuccess) e = put(&t.eout_L, c->host.e_out_L);
    if (e == cudaSuccess) e = put(&t.eout_M, c->host.e_out_M);
    for (int k = 0; k < 3 && e == cudaSuccess; ++k) e = put(&t.H[k], c->host.H[k]);
    if (e != cudaSuccess) {
        free_tables(t);  // a partial set is retried from scratch on the next call
        free_offsets(c);
        return cuda_fail(c, e, "table upload");
    }
    t.ready = true;
    return SFMM_OK;
}

// arrays laid end to end for one allocation and one copy; add() returns an offset
struct Blob {
    std::vector<unsigned char> bytes;
    template <class T>
    size_t add(const std::vector<T> &v)
    {
        const size_t at = (bytes.size() + 255) & ~size_t(255);
        bytes.resize(at + v.size() * sizeof(T));
        if (!v.empty()) std::memcpy(&bytes[at], v.data(), v.size() * sizeof(T));
        return at;
    }
};

// edge factors in the arithmetic's form
size_t add_edges(Blob &b, Arith a, const std::vector<double> &e, size_t ne)
{
    if (a == Arith::F64) return b.add(fx_edges(e, ne));
    std::vector<float> v;
    for (size_t i = 0; i < ne; ++i) {
        v.push_back((float)e[i]);
        if (a == Arith::FFQ) v.push_back((float)(e[i] - (double)v.back()));
    }
    return b.add(v);
}

// the tables of one group size: swap coefficients of wsize bytes per woff unit
template <class T>
void add_group(Blob &b, FxDevTables &t, size_t (&at)[4], const T &h, int P, size_t wsize)
{
    at[0] = b.add(h.W);
    for (int k = 0; k < 3; ++k) at[1 + k] = b.add(h.H[k]);
    t.wend.assign(P + 1, (int)(h.W.size() * sizeof(h.W[0])));
    for (int n = 0; n < P; ++n) t.wend[n] = (int)(h.woff[n] * wsize);
    t.hbytes = (int)(h.H[0].size() * sizeof(h.H[0][0]));
    t.P = P;
}

// tables of the 60-bit fixed-point (F64), the FP32 or the split kernel (FFQ):
// orders up to 32, both group sizes
int ensure_fx(sfmm_context *c, Arith a)
{
    ArithTables &t = c->fxt[(int)a];
    if (t.mem) return SFMM_OK;
    const int P = std::min(c->P, 32);
    cudaError_t e;
    try {
        Blob b;
        const std::vector<double> *ev[4] = {&c->host.e_in_M, &c->host.e_in_L, &c->host.e_out_L, &c->host.e_out_M};
        size_t edge[4], at[2][4];
        for (int k = 0; k < 4; ++k) edge[k] = add_edges(b, a, *ev[k], (size_t)P * (P + 1) / 2);
        for (int k = 0; k < 2; ++k) {
            const int G = k ? 8 : 4;
            if (a == Arith::F32) add_group(b, t.group[k], at[k], build_f32_tables(c->host, G, P), P, sizeof(float));
            else if (a == Arith::F64) add_group(b, t.group[k], at[k], build_fx_tables(c->host, G, P), P, 2 * sizeof(int32_t));
            else add_group(b, t.group[k], at[k], build_split_tables(c->host, G, P), P, 2 * sizeof(int32_t));
        }
        e = put(&t.mem, b.bytes);
        const unsigned char *mem = static_cast<const unsigned char *>(t.mem);
        for (int k = 0; k < 4 && e == cudaSuccess; ++k) t.edge[k] = mem + edge[k];
        for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
            t.group[k].W = mem + at[k][0];
            for (int op = 0; op < 3; ++op) t.group[k].H[op] = mem + at[k][1 + op];
        }
    } catch (const std::bad_alloc &) {
        free_arith(t);
        return fail(c, SFMM_OOM, "operator tables");
    }
    if (e != cudaSuccess) {
        free_arith(t);  // retried from scratch on the next call
        return cuda_fail(c, e, "table upload");
    }
    return SFMM_OK;
}

}  // namespace

// Split precision keeps its 1e-7 contract (orthonormal basis) with the
// fixed-point rotations for M2L and L2L up to order 28 and M2M up to order
// 18.  Past that the rotation method's own error growth with the degree
// (about 1.35x per degree for M2M, in every arithmetic) pushes 30-bit
// mantissas above 1e-7, and the batch runs as SFMM_SPLIT_FF instead.
constexpr int kFixedM2MOrder = 18;

// Everything that launches of this arithmetic read on this context, whatever
// their order bound and group size, on its first use: a call of the same
// arithmetic recorded in a stream capture later allocates nothing.  Split's
// M2M above kFixedM2MOrder reads the FP64 kernel's tables.
int ensure_tables(sfmm_context *c, Arith a)
{
    if (is_tc(a)) {
        const int mode = tc_mode(a);
        if (c->tc[mode]) return SFMM_OK;
        cudaError_t e = tc_prepare(&c->tc[mode], mode, c->host);
        if (e != cudaSuccess) return cuda_fail(c, e, "tensor-core table upload");
        return SFMM_OK;
    }
    if (a == Arith::FF) return SFMM_OK;  // above its orders: no kernel
    int st = ensure_fx(c, a);
    if (st == SFMM_OK && a == Arith::FFQ && c->P > kFixedM2MOrder) st = ensure_fx(c, Arith::F64);
    if (st == SFMM_OK && a == Arith::F64 && c->P > 32) st = ensure_high(c);
    return st;
}

int arith_of(sfmm_context *c, int precision, Arith *out)
{
    if (precision == SFMM_PLAIN) {
        *out = c->dtype == SFMM_F64 ? Arith::F64 : Arith::F32;
        return SFMM_OK;
    }
    if (precision == SFMM_SPLIT || precision == SFMM_SPLIT_FF) {
        if (c->dtype != SFMM_F64)
            return fail(c, SFMM_UNSUPPORTED, "split precision needs an FP64 context (FP64 accumulation targets)");
        *out = precision == SFMM_SPLIT ? Arith::FFQ : Arith::FF;
        return SFMM_OK;
    }
    if (precision == SFMM_TC_TF32 || precision == SFMM_TC_BF16 || precision == SFMM_TC_BF16X6) {
        if (c->dtype != SFMM_F64)
            return fail(c, SFMM_UNSUPPORTED, "tensor-core precision needs an FP64 context (FP64 accumulation targets)");
        *out = precision == SFMM_TC_TF32 ? Arith::TC32 : (precision == SFMM_TC_BF16 ? Arith::TC16 : Arith::TC16X6);
        return SFMM_OK;
    }
    return fail(c, SFMM_INVALID_ARG, "unknown precision mode %d", precision);
}

// The tensor-core kernel holds a tile's expansions in tensor memory up to
// order 16; batches with a larger order bound run the split kernel.
Arith resolve_mode(Arith a, int op, int Pbound)
{
    if (is_tc(a) && Pbound > tc_max_order()) a = Arith::FFQ;
    if (a == Arith::FFQ && op == SFMM_M2M && Pbound > kFixedM2MOrder) a = Arith::FF;
    return a;
}

// SFMM_SPLIT_FF runs the FP64 kernel, whose 60-bit fixed point rounds less than
// float-float did (M2L P=16 2e-15 against 7e-14) and is as fast or faster but for
// some batches: M2L in M/s, fixed point / float-float, P=6 592 / 499, P=16 86.5 /
// 77.8, P=20 47.7 / 44.8, P=22 30.9 / 33.2, P=24 22.1 / 23.5, P=26 15.6 / 17.9,
// P=28 13.5 / 13.5; FMM pass at P=12 31.5 / 35.4 ms; one translation at P=12 68 /
// 56 us; orders 4 to 24 in no order 20.5 / 27.5 (plans sort them).  No shape of
// the fixed-point kernel closes those, and its accuracy is what the mode has now.
// Orders above kMaxFloatOrder, which the mode never took, keep Arith::FF and
// are refused by prepare_launch.
Arith resolve_arith(Arith a, int op, int Pbound)
{
    a = resolve_mode(a, op, Pbound);
    return a == Arith::FF && Pbound <= kMaxFloatOrder ? Arith::F64 : a;
}

int prepare_launch(sfmm_context *c, int op, Arith a, int Pbound, LaunchShape *shape)
{
    const Arith mode = resolve_mode(a, op, Pbound);
    a = resolve_arith(a, op, Pbound);
    if (Pbound < 1) Pbound = 1;
    std::lock_guard<std::mutex> lk(c->setup_mtx);
    if (is_tc(a)) {  // one 128-thread CTA per SM, one translation per thread
        int st = ensure_tables(c, a);
        if (st) return st;
        if (shape) {
            *shape = LaunchShape{};
            shape->G = 1;
            shape->acc = 1;
            shape->TS = 128;
            shape->threads = 128;
            shape->blocks_per_sm = 1;
        }
        return SFMM_OK;
    }
    if (a != Arith::F64 && Pbound > kMaxFloatOrder)
        return fail(c, SFMM_UNSUPPORTED, "order %d exceeds %d, the limit of FP32-range arithmetic", Pbound, kMaxFloatOrder);
    const auto key = std::make_tuple(op, (int)mode, Pbound);
    auto it = c->shapes.find(key);
    if (it == c->shapes.end()) it = c->shapes.emplace(key, best_shape(a, Pbound, default_group(a, Pbound))).first;
    if (shape) *shape = it->second;
    if (it->second.acc == 0)
        return fail(c, SFMM_UNSUPPORTED, "order %d exceeds the GPU kernels' limit %d", Pbound, kMaxKernelOrder);
    return ensure_tables(c, a);
}

void set_shape(sfmm_context *c, std::tuple<int, int, int> key, const LaunchShape *s)
{
    std::lock_guard<std::mutex> lk(c->setup_mtx);
    if (s) c->shapes[key] = *s;
    else c->shapes.erase(key);
}

const void *device_view(sfmm_context *c, const void *host)
{
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (at.type == cudaMemoryTypeHost && at.devicePointer && at.device == c->device) return at.devicePointer;
    if (at.type == cudaMemoryTypeUnregistered && c->pageable_access) return host;
    return nullptr;
}

// The launch itself: validated arguments, device pointers.
int run_batch(sfmm_context *c, cudaStream_t stream, int op, Arith a, int Pbound, long long n, const void *src,
              long long sstride, long long nsrc, const uint32_t *sidx, void *dst, long long dstride, long long ndst,
              const uint32_t *tidx, const uint32_t *pin, const uint32_t *pout, const double *shift,
              const uint32_t *perm, int flags, long long nidx, const unsigned long long *src_ptr,
              const unsigned long long *dst_ptr, bool in_hbm, const WorkList *wl, const LaunchShape *shape)
{
    if (n == 0) return SFMM_OK;
    static const char *const kName[3] = {"sfmm m2m launch", "sfmm m2l launch", "sfmm l2l launch"};
    Range range(kName[(op >= SFMM_M2M && op <= SFMM_L2L) ? op - SFMM_M2M : 1]);
    LaunchShape s;
    int st = prepare_launch(c, op, a, Pbound, &s);
    if (st) return st;
    a = resolve_arith(a, op, Pbound);
    if (Pbound < 1) Pbound = 1;
    if (shape && !is_tc(a)) s = *shape;
    KParams p{};
    p.op = op;
    p.P = Pbound;
    p.Ptab = c->P;
    p.n = n;
    p.src = src;
    p.sstride = sstride;
    p.nsrc = nsrc;
    p.sidx = sidx;
    p.dst = dst;
    p.dstride = dstride;
    p.ndst = ndst;
    p.tidx = tidx;
    p.status = c->d_status;
    p.pin = pin;
    p.pout = pout;
    p.shift = shift;
    p.perm = perm;
    p.nidx = nidx < 0 ? n : nidx;
    p.src_ptr = src_ptr;
    p.dst_ptr = dst_ptr;
    p.atomic = (flags & SFMM_TARGETS_REPEAT) ? 1 : 0;
    p.in_hbm = in_hbm ? 1 : 0;
    if (wl) {
        if (is_tc(a)) return fail(c, SFMM_UNSUPPORTED, "work lists run the split and plain kernels");
        p.work = wl->work;
        p.work_counter = wl->counter;
        p.nwork = wl->n;
    }
    if (is_tc(a)) {
        cudaError_t e = launch_translate_tc(p, c->tc[tc_mode(a)], c->num_sms, stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "tensor-core translation kernel launch");
        c->launches++;
        return SFMM_OK;
    }
    if (s.fx) {
        const FxDevTables &t = c->fxt[(int)a].group[s.G == 8];
        p.W = t.W;
        p.Ptab = t.P;
        p.ein = c->fxt[(int)a].edge[op == SFMM_L2L ? 1 : 0];
        p.eout = c->fxt[(int)a].edge[op == SFMM_M2M ? 3 : 2];
        p.H = t.H[op];
        p.wbytes = t.wend[Pbound];
        p.hbytes = t.P == Pbound ? t.hbytes : 0;  // a smaller bound reads parts of every row
    } else {
        const DevTables &t = c->tab;
        p.W = t.W;
        p.woff = c->d_woff;
        p.hoff = c->d_hoff;
        p.rowpad = c->host.pad;
        p.ein = (op == SFMM_L2L) ? t.ein_L : t.ein_M;
        p.eout = (op == SFMM_M2M) ? t.eout_M : t.eout_L;
        p.H = t.H[op];
    }
    p.spad = s.spad;
    p.TS = s.TS;
    long long tiles = wl ? wl->n : (n + s.TS - 1) / s.TS;
    long long grid = (long long)c->num_sms * s.blocks_per_sm;
    if (grid > tiles) grid = tiles;
    if (grid < 1) return fail(c, SFMM_CUDA_ERROR, "no launch shape runs order %d (G %d, %d translations per CTA)",
                              Pbound, s.G, s.TS);
    if (a != Arith::F64 && s.spad > kDegreeTableSize)
        return fail(c, SFMM_UNSUPPORTED, "buffer of %d slots above the FP32-range kernels' degree table", s.spad);
    if (wl) {  // the tile descriptor's two words after the meta arrays
        s.smem += 8;
        if (s.smem > 232448) return fail(c, SFMM_UNSUPPORTED, "work-list launch above the shared-memory limit");
    }
    cudaError_t e = launch_translate(a, p, s, (int)grid, stream);
    if (e != cudaSuccess)
        return fail(c, SFMM_CUDA_ERROR, "translation kernel launch (order %d, G %d, %d per CTA, %zu B shared, grid %lld): %s",
                    Pbound, s.G, s.TS, s.smem, grid, cudaGetErrorString(e));
    c->launches++;
    return SFMM_OK;
}

}  // namespace sfmm

namespace sfmm {

LaunchShape translate_shape(Arith a, int P, int G, int ts)
{
    LaunchShape s;
    const int per_warp = 32 / G;  // translations per warp
    if (P < 1 || P > kMaxKernelOrder || ts < per_warp || ts % per_warp || G * ts > 256) return s;
    if ((G == 32) != (P > 32)) return s;  // one warp per translation exactly for orders above 32
    int acc = (P + G - 1) / G;
    if (G == 4) acc = acc <= 2 ? acc : (acc <= 4 ? 4 : (acc <= 6 ? 6 : 8));
    if (G == 32) acc = acc <= 2 ? 2 : 3;
    s.fx = G != 32;
    if (a == Arith::F64 || a == Arith::F32) {
        // one part of an element per lane, rows in steps of G/2.  FP64 runs
        // four threads per translation only up to order 16 (more rows than
        // their registers hold: above, a request for 4 runs 8)
        if (G != 32) {
            if (P > 16 && G == 4 && a == Arith::F64) {
                G = 8;
                ts /= 2;
                if (ts < 32 / G || ts % (32 / G)) return LaunchShape{};
            }
            if (G * ts > kFxThreads) return LaunchShape{};
            acc = (P + G / 2 - 1) / (G / 2);
            if (a == Arith::F32) acc = acc <= 4 ? 4 : acc <= 6 ? 6 : acc <= 8 ? 8 : acc <= 10 ? 10 : 14;
            else acc = G == 4 ? (acc <= 4 ? 4 : acc <= 6 ? 6 : 8) : (acc + 1) / 2 * 2;
        }
    } else if (G == 32) {
        return LaunchShape{};
    }
    s.G = G;
    s.acc = acc;
    int scap = P * (P + 1) + 4;  // room for the swap loops' zero-coefficient reads past the last row
    // Translation stride in shared memory.  The swap and z loops read one or
    // two slots per translation, broadcast to its group; the per-element
    // stages touch G consecutive slots per translation.  With 8 translations
    // per warp (G = 4) bases 4 banks apart keep the broadcasts conflict-free;
    // with 4 per warp (G = 8) bases 8 banks apart keep both patterns at the
    // minimum number of wavefronts.
    const int mod = esize(a) == 8 ? 16 : 32;
    const int want = esize(a) == 8 ? (G == 8 ? 4 : 2) : (G == 8 ? 8 : 4);
    s.spad = scap + ((want - scap) % mod + mod) % mod;
    s.TS = ts;
    s.threads = G * ts;
    s.smem = (size_t)ts * s.spad * esize(a) + 5 * sizeof(uint32_t) * ts +
             (s.fx && a != Arith::FFQ && a != Arith::FF ? ts * sizeof(FxGeo) : 0);
    if (s.smem > 232448) return LaunchShape{};
    return s;
}

// Threads per translation by default: one warp above order 32; below, 4 or
// 8 from a sweep on GB300 (M2L, uniform orders 2..32, both group sizes): 8
// threads pay off once the per-translation buffers limit the SM to a few
// warps and the group's own arithmetic is cheap enough to leave latency
// exposed (split from 14; FP32 from 15: M2L at P=14 338 M/s with 4 and 311 with 8,
// at P=16 251 and 266, at P=20 136 and 145).  FP64 (60-bit fixed point)
// from 13, where four threads need more rows than fit the registers of a full
// SM: M2L at P=12 189 M/s with 4 and 150 with 8, at P=13 89 and 125.
int default_group(Arith a, int P)
{
    if (P > 32) return 32;
    switch (a) {
    case Arith::F64: return P >= 13 ? 8 : 4;
    case Arith::F32: return P >= 15 ? 8 : 4;
    case Arith::FFQ: return P >= 14 ? 8 : 4;
    }
    return 4;
}

// The tile size that keeps the most threads resident per SM (shared memory
// and registers permitting) for G threads per translation; ties go to the
// larger tile (fewer CTAs), or to the smaller one with small_tiles (shorter
// waits at the tile barriers).
LaunchShape best_shape(Arith a, int P, int G, bool small_tiles, int min_threads)
{
    // By default CTAs of at least four warps: one-warp tiles can hold a few
    // more threads per SM at high orders, but ran up to 40% slower on GB300
    // (split M2L P=22: 1 976 CTAs of 32 threads, instruction-fetch stalls and
    // a lower L1 hit rate for the tables); smaller CTAs when no larger tile
    // fits, or when sfmm_tune measures them faster (split P=27: +6%).  The
    // 60-bit kernel also takes two warps (three above order 22) where they
    // hold an eighth more threads: M2L P=21 1.72 ms (2.01 with four warps), P=24
    // 2.01 (2.18), P=30 2.22 (2.82), while with equal numbers they are level
    // (P=22, 23, 26) or four win (P=20 1.60, two 1.77).  One- and two-warp CTAs
    // would give P=24 1.77 and 1.85, but only while all of them run in step: a
    // launch of orders 4 to 24 in no order, whose warps wait for instructions,
    // takes 4.30 and 2.78 ms with them, 2.17 with three and 2.00 with four.
    const int few = a == Arith::F64 ? (P <= 22 ? 64 : 96) : 32;
    LaunchShape best[2];
    long most[2] = {0, 0};
    for (int k = 0; k < 2; ++k)
        for (int ts = 256 / G; ts >= 32 / G; ts -= 32 / G) {
            LaunchShape s = translate_shape(a, P, G, ts);
            if (!s.acc || s.threads < (k ? (best[0].acc ? few : 32) : min_threads)) continue;
            s.blocks_per_sm = translate_blocks_per_sm(a, s);
            const long th = (long)s.blocks_per_sm * s.threads;
            if (th > 0 && (th > most[k] || (small_tiles && th == most[k]))) {
                most[k] = th;
                best[k] = s;
            }
        }
    if (!best[0].acc || (a == Arith::F64 && 8 * most[1] >= 9 * most[0])) return best[1];
    return best[0];
}

cudaError_t launch_translate_64(const KParams &, const LaunchShape &, int, cudaStream_t);
cudaError_t launch_translate_fx(const KParams &, const LaunchShape &, int, cudaStream_t);
int occupancy_fx64(const LaunchShape &);
cudaError_t launch_translate_32(const KParams &, const LaunchShape &, int, cudaStream_t);
cudaError_t launch_translate_ffq(const KParams &, const LaunchShape &, int, cudaStream_t);
int occupancy_64(const LaunchShape &);
int occupancy_32(const LaunchShape &);
int occupancy_ffq(const LaunchShape &);

cudaError_t launch_translate(Arith a, const KParams &p, const LaunchShape &s, int grid, cudaStream_t st)
{
    switch (a) {
    case Arith::F64: return s.fx ? launch_translate_fx(p, s, grid, st) : launch_translate_64(p, s, grid, st);
    case Arith::F32: return launch_translate_32(p, s, grid, st);
    case Arith::FFQ: return launch_translate_ffq(p, s, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

int translate_blocks_per_sm(Arith a, const LaunchShape &s)
{
    switch (a) {
    case Arith::F64: return s.fx ? occupancy_fx64(s) : occupancy_64(s);
    case Arith::F32: return occupancy_32(s);
    case Arith::FFQ: return occupancy_ffq(s);
    default: return 1;  // Arith::FF above its orders: a shape to pin, no kernel
    }
}

}  // namespace sfmm

extern "C" {

const char *sfmm_status_string(int s)
{
    switch (s) {
    case SFMM_OK: return "ok";
    case SFMM_INVALID_ARG: return "invalid argument";
    case SFMM_ORDER_RANGE: return "order out of range";
    case SFMM_OVERFLOW: return "order too large for the floating-point type";
    case SFMM_DIM_MISMATCH: return "dimension mismatch";
    case SFMM_OOM: return "out of memory";
    case SFMM_CUDA_ERROR: return "CUDA error";
    case SFMM_UNSUPPORTED: return "unsupported";
    default: return "unknown status";
    }
}

int sfmm_create(sfmm_context **out, int dtype, size_t P, int device)
{
    if (!out) return SFMM_INVALID_ARG;
    *out = nullptr;
    if (dtype != SFMM_F32 && dtype != SFMM_F64) return SFMM_INVALID_ARG;
    if (P == 0) return SFMM_INVALID_ARG;
    if ((dtype == SFMM_F32 && P > (size_t)kMaxFloatOrder) || (dtype == SFMM_F64 && P > 86)) return SFMM_OVERFLOW;
    sfmm_context *c = new (std::nothrow) sfmm_context;
    if (!c) return SFMM_OOM;
    c->dtype = dtype;
    c->P = (int)P;
    c->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device) == cudaSuccess)
            c->pageable_access = v != 0;
    }
    if (e != cudaSuccess) {
        delete c;
        return SFMM_CUDA_ERROR;
    }
    try {
        c->host = build_tables((int)P);
    } catch (const std::bad_alloc &) {
        delete c;
        return SFMM_OOM;
    }
    if (cudaMalloc(&c->d_status, sizeof(int)) != cudaSuccess || cudaMemset(c->d_status, 0, sizeof(int)) != cudaSuccess) {
        if (c->d_status) cudaFree(c->d_status);
        delete c;
        return SFMM_CUDA_ERROR;
    }
    *out = c;
    return SFMM_OK;
}

void sfmm_destroy(sfmm_context *c)
{
    if (!c) return;
    cudaSetDevice(c->device);
    free_tables(c->tab);
    for (auto &t : c->tc) tc_release(t);
    for (auto &t : c->fxt) free_arith(t);
    for (int k = 0; k < 3; ++k) {
        c->d_src[k].release();
        c->d_dst[k].release();
        c->d_meta[k].release();
        c->d_shift[k].release();
        if (c->pipe[k]) cudaStreamDestroy(c->pipe[k]);
    }
    c->d_work.release();
    c->d_eval.release();
    c->d_eval_grad.release();
    if (c->d_status) cudaFree(c->d_status);
    free_offsets(c);
    c->h_src.release();
    c->h_dst.release();
    c->h_meta.release();
    c->h_shift.release();
    delete c;
}

size_t sfmm_order(const sfmm_context *c) { return c ? (size_t)c->P : 0; }
int sfmm_data_type(const sfmm_context *c) { return c ? c->dtype : -1; }
const char *sfmm_last_error(const sfmm_context *c) { return c ? c->err.c_str() : "null context"; }
uint64_t sfmm_launch_count(const sfmm_context *c) { return c ? c->launches.load() : 0; }

int sfmm_host_table(size_t P, int which, int n, double *out, size_t cap, size_t *count)
{
    if (P == 0 || P > 86 || !count) return SFMM_INVALID_ARG;
    HostTables t;
    try {
        t = build_tables((int)P);
    } catch (const std::bad_alloc &) {
        return SFMM_OOM;
    }
    std::vector<double> v;
    if (which == 0 || which == 1) {  // dense W_R / W_I of degree n, row-major (i, j)
        if (n < 0 || n >= (int)P) return SFMM_INVALID_ARG;
        const int d = n + 1;
        for (int i = 0; i < d; ++i)
            for (int j = 0; j < d; ++j) v.push_back(w_entry(t, n, which, i, j));
    } else if (which >= 2 && which <= 4) {  // dense H_m (n', k) of op which-2, row-major, m = n
        const int m = n, L = (int)P - m;
        if (m < 0 || m >= (int)P) return SFMM_INVALID_ARG;
        const int HR = hrows(L, t.pad);
        for (int a = 0; a < L; ++a)
            for (int k = 0; k < L; ++k) v.push_back(t.H[which - 2][t.hoff[m] + (size_t)k * HR + a]);
    } else if (which >= 5 && which <= 8) {  // edge factors
        const std::vector<double> *e[] = {&t.e_in_M, &t.e_in_L, &t.e_out_L, &t.e_out_M};
        v = *e[which - 5];
    } else {
        return SFMM_INVALID_ARG;
    }
    *count = v.size();
    if (out) std::memcpy(out, v.data(), sizeof(double) * std::min(cap, v.size()));
    return SFMM_OK;
}

int sfmm_set_stream(sfmm_context *c, void *stream)
{
    if (!c) return SFMM_INVALID_ARG;
    c->stream = (cudaStream_t)stream;
    return SFMM_OK;
}

int sfmm_set_group(sfmm_context *c, int precision, size_t order_bound, int group)
{
    if (!c) return SFMM_INVALID_ARG;
    std::lock_guard<std::mutex> lk(c->mtx);
    Arith a;
    int st = arith_of(c, precision, &a);
    if (st) return st;
    if (order_bound > (size_t)c->P) return fail(c, SFMM_ORDER_RANGE, "order bound %zu exceeds the context order %d", order_bound, c->P);
    const int Pb = order_bound ? (int)order_bound : c->P;
    if (is_tc(resolve_arith(a, SFMM_M2L, Pb)))
        return fail(c, SFMM_UNSUPPORTED, "the tensor-core kernel runs one thread per translation");
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, SFMM_CUDA_ERROR, "cannot select device %d", c->device);
    LaunchShape s[3];
    for (int op = SFMM_M2M; op <= SFMM_L2L; ++op) {  // every operator at this order
        s[op - SFMM_M2M] = best_shape(resolve_arith(a, op, Pb), Pb, group);
        if (!s[op - SFMM_M2M].acc)
            return fail(c, SFMM_INVALID_ARG, "no kernel runs %d threads per translation at order %d", group, Pb);
    }
    std::lock_guard<std::mutex> lk2(c->setup_mtx);
    for (int op = SFMM_M2M; op <= SFMM_L2L; ++op)
        if ((st = ensure_tables(c, resolve_arith(a, op, Pb)))) return st;  // before a capture may launch it
    for (int op = SFMM_M2M; op <= SFMM_L2L; ++op)
        c->shapes[std::make_tuple(op, (int)resolve_mode(a, op, Pb), Pb)] = s[op - SFMM_M2M];
    return SFMM_OK;
}

int sfmm_tune(sfmm_context *c, int op, int precision, size_t order_bound, size_t n, int *group, double *rate)
{
    if (!c) return SFMM_INVALID_ARG;
    std::lock_guard<std::mutex> lk(c->mtx);
    if (op < SFMM_M2M || op > SFMM_L2L) return fail(c, SFMM_INVALID_ARG, "unknown operation %d", op);
    Arith a;
    int st = arith_of(c, precision, &a);
    if (st) return st;
    if (order_bound > (size_t)c->P) return fail(c, SFMM_ORDER_RANGE, "order bound %zu exceeds the context order %d", order_bound, c->P);
    if (n == 0 || n > (size_t)1 << 24) return fail(c, SFMM_INVALID_ARG, "tuning sample of %zu translations", n);
    const int Pb = order_bound ? (int)order_bound : c->P;
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, SFMM_CUDA_ERROR, "cannot select device %d", c->device);
    const size_t S = (size_t)Pb * (Pb + 1), es = c->dtype == SFMM_F64 ? 8 : 4;
    // synthetic batch: constant coefficients, orders Pb, shifts of length
    // 2.5 in varied directions (the kernels' cost does not depend on values)
    std::vector<uint32_t> ord(n, (uint32_t)Pb);
    std::vector<double> sh(3 * n);
    for (size_t i = 0; i < n; ++i) {
        const double t = 0.7 * (double)i, u = 0.3 + 2.4 * (double)(i % 97) / 97.0;
        sh[3 * i] = 2.5 * std::sin(u) * std::cos(t);
        sh[3 * i + 1] = 2.5 * std::sin(u) * std::sin(t);
        sh[3 * i + 2] = 2.5 * std::cos(u);
    }
    void *src = nullptr, *dst = nullptr, *meta = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    auto cleanup = [&] {
        if (src) cudaFree(src);
        if (dst) cudaFree(dst);
        if (meta) cudaFree(meta);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
    };
    cudaError_t e;
    if ((e = cudaMalloc(&src, n * S * es)) != cudaSuccess || (e = cudaMalloc(&dst, n * S * es)) != cudaSuccess ||
        (e = cudaMalloc(&meta, n * (2 * sizeof(uint32_t) + 3 * sizeof(double)))) != cudaSuccess) {
        cleanup();
        return e == cudaErrorMemoryAllocation ? fail(c, SFMM_OOM, "tuning buffers") : cuda_fail(c, e, "tuning buffers");
    }
    double *d_shift = static_cast<double *>(meta);
    uint32_t *d_ord = reinterpret_cast<uint32_t *>(d_shift + 3 * n);
    cudaStream_t stream = c->stream;
    if ((e = cudaMemsetAsync(src, 0x3e, n * S * es, stream)) != cudaSuccess ||
        (e = cudaMemsetAsync(dst, 0, n * S * es, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(d_shift, sh.data(), 3 * n * sizeof(double), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(d_ord, ord.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaEventCreate(&e0)) != cudaSuccess || (e = cudaEventCreate(&e1)) != cudaSuccess) {
        cleanup();
        return cuda_fail(c, e, "tuning setup");
    }
    const Arith mode = resolve_mode(a, op, Pb);
    a = resolve_arith(a, op, Pb);
    if (is_tc(a)) {  // one launch shape: time it
        float ms = 0;
        for (int rep = 0; rep < 2 && st == SFMM_OK; ++rep) {
            if (rep == 1 && (e = cudaEventRecord(e0, stream)) != cudaSuccess) break;
            for (int k = 0; k < (rep ? 3 : 1) && st == SFMM_OK; ++k)
                st = run_batch(c, stream, op, a, Pb, (long long)n, src, (long long)S, (long long)n, nullptr, dst,
                               (long long)S, (long long)n, nullptr, d_ord, d_ord, d_shift, nullptr, 0);
            if (rep == 1 && (e = cudaEventRecord(e1, stream)) != cudaSuccess) break;
        }
        if (st == SFMM_OK && e == cudaSuccess && (e = cudaEventSynchronize(e1)) == cudaSuccess)
            e = cudaEventElapsedTime(&ms, e0, e1);
        cleanup();
        if (st != SFMM_OK) return st;
        if (e != cudaSuccess) return cuda_fail(c, e, "tuning run");
        if (group) *group = 1;
        if (rate) *rate = ms > 0 ? 3.0 * (double)n / (ms * 1e-3) : 0.0;
        return SFMM_OK;
    }
    const auto key = std::make_tuple(op, (int)mode, Pb);
    LaunchShape best;
    double best_rate = 0;
    // candidates: every group size that runs at this order, each with the
    // largest and the smallest full-occupancy tile, among CTAs of four warps
    // or more and among all tiles (distinct shapes only)
    LaunchShape cands[12];
    int ncand = 0;
    for (int G : {4, 8, 32})
        for (int min_threads : {128, 32})
            for (bool small : {false, true}) {
                const LaunchShape s = best_shape(a, Pb, G, small, min_threads);
                bool seen = !s.acc;
                for (int k = 0; k < ncand && !seen; ++k) seen = cands[k].G == s.G && cands[k].TS == s.TS;
                if (!seen) cands[ncand++] = s;
            }
    for (int ci = 0; ci < ncand; ++ci) {
        const LaunchShape s = cands[ci];
        set_shape(c, key, &s);
        float ms = 0;
        for (int rep = 0; rep < 2 && st == SFMM_OK; ++rep) {  // warm-up, then timed
            if (rep == 1 && (e = cudaEventRecord(e0, stream)) != cudaSuccess) break;
            for (int k = 0; k < (rep ? 3 : 1) && st == SFMM_OK; ++k)
                st = run_batch(c, stream, op, mode, Pb, (long long)n, src, (long long)S, (long long)n, nullptr, dst,
                               (long long)S, (long long)n, nullptr, d_ord, d_ord, d_shift, nullptr, 0);
            if (rep == 1 && (e = cudaEventRecord(e1, stream)) != cudaSuccess) break;
        }
        if (st == SFMM_OK && e == cudaSuccess && (e = cudaEventSynchronize(e1)) == cudaSuccess)
            e = cudaEventElapsedTime(&ms, e0, e1);
        if (st != SFMM_OK || e != cudaSuccess) {
            set_shape(c, key, nullptr);
            cleanup();
            return st != SFMM_OK ? st : cuda_fail(c, e, "tuning run");
        }
        const double r = ms > 0 ? 3.0 * (double)n / (ms * 1e-3) : 0.0;
        if (r > best_rate) {
            best_rate = r;
            best = s;
        }
    }
    cleanup();
    if (!best.acc) {
        set_shape(c, key, nullptr);
        return fail(c, SFMM_UNSUPPORTED, "no kernel for order %d", Pb);
    }
    set_shape(c, key, &best);
    {
        std::lock_guard<std::mutex> lk2(c->setup_mtx);
        c->tuned.insert(std::make_tuple(op, (int)mode, Pb));
    }
    if (group) *group = best.G;
    if (rate) *rate = best_rate;
    return SFMM_OK;
}

int sfmm_translate_device(sfmm_context *c, int op, int precision, size_t n, const void *src, size_t src_stride,
                          size_t src_count, const uint32_t *src_index, void *dst, size_t dst_stride,
                          size_t dst_count, const uint32_t *dst_index, const uint32_t *p_in, const uint32_t *p_out,
                          const double *shift, const uint32_t *order, int flags, size_t order_bound)
{
    if (!c) return SFMM_INVALID_ARG;
    if (op < SFMM_M2M || op > SFMM_L2L) return fail(c, SFMM_INVALID_ARG, "unknown operator %d", op);
    Arith a;
    int st = arith_of(c, precision, &a);
    if (st) return st;
    if (n == 0) return SFMM_OK;
    if (n > 0xffffffffull) return fail(c, SFMM_INVALID_ARG, "batch larger than 2^32 translations");
    if (!src || !dst || !p_in || !p_out || !shift)
        return fail(c, SFMM_INVALID_ARG, "null device pointer in batch");
    size_t bound = order_bound ? order_bound : (size_t)c->P;
    if (bound > (size_t)c->P) return fail(c, SFMM_ORDER_RANGE, "order bound %zu exceeds operator order %d", bound, c->P);
    if (src_stride < bound * (bound + 1) || dst_stride < bound * (bound + 1))
        return fail(c, SFMM_INVALID_ARG, "expansion stride smaller than P(P+1) for the order bound");
    cudaSetDevice(c->device);
    return run_batch(c, c->stream, op, a, (int)bound, (long long)n, src, (long long)src_stride,
                     (long long)src_count, src_index, dst, (long long)dst_stride, (long long)dst_count, dst_index,
                     p_in, p_out, shift, order, flags);
}

int sfmm_device_status(sfmm_context *c, int *flags)
{
    if (!c || !flags) return SFMM_INVALID_ARG;
    cudaSetDevice(c->device);
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "stream synchronise");
    int v = 0;
    e = cudaMemcpy(&v, c->d_status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemset(c->d_status, 0, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(c, e, "status read");
    *flags = v;
    return SFMM_OK;
}

int sfmm_bucket_by_order(sfmm_context *c, size_t n, const uint32_t *p_in, const uint32_t *p_out, uint32_t *order)
{
    if (!c) return SFMM_INVALID_ARG;
    Range range("sfmm bucket");
    if (n == 0) return SFMM_OK;
    if (!p_in || !p_out || !order) return fail(c, SFMM_INVALID_ARG, "null device pointer");
    if (n > 0xffffffffull) return fail(c, SFMM_INVALID_ARG, "batch larger than 2^32 - 1 translations");
    cudaSetDevice(c->device);
    cudaError_t e = c->d_work.ensure(bucket_work_words(c->P) * sizeof(uint32_t));
    if (e != cudaSuccess) return cuda_fail(c, e, "bucket workspace");
    e = launch_bucket((long long)n, p_in, p_out, order, (uint32_t *)c->d_work.p, c->P, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "bucket kernels");
    c->launches += 3;
    return SFMM_OK;
}

int sfmm_p2x_device(sfmm_context *c, int kind, size_t nexp, size_t nq, const double *charge, const double *pos,
                    const double *centre, void *out, size_t out_stride)
{
    if (!c) return SFMM_INVALID_ARG;
    Range range("sfmm p2m/p2l");
    if (kind != 0 && kind != 1) return fail(c, SFMM_INVALID_ARG, "kind must be 0 (P2M) or 1 (P2L)");
    if (nexp == 0) return SFMM_OK;
    if (!charge || !pos || !centre || !out) return fail(c, SFMM_INVALID_ARG, "null device pointer");
    if (out_stride < (size_t)c->P * (c->P + 1)) return fail(c, SFMM_INVALID_ARG, "stride smaller than P(P+1)");
    cudaSetDevice(c->device);
    cudaError_t e = launch_p2x(c->dtype == SFMM_F64, kind, c->P, (long long)nexp, (long long)nq, nullptr, charge,
                               pos, centre, out, (long long)out_stride, c->num_sms, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "P2M/P2L kernel");
    c->launches++;
    return SFMM_OK;
}

int sfmm_p2x_ragged_device(sfmm_context *c, int kind, size_t nexp, const uint32_t *offset, const double *charge,
                           const double *pos, const double *centre, void *out, size_t out_stride)
{
    if (!c) return SFMM_INVALID_ARG;
    Range range("sfmm p2m/p2l");
    if (kind != 0 && kind != 1) return fail(c, SFMM_INVALID_ARG, "kind must be 0 (P2M) or 1 (P2L)");
    if (nexp == 0) return SFMM_OK;
    if (!offset || !charge || !pos || !centre || !out) return fail(c, SFMM_INVALID_ARG, "null device pointer");
    if (out_stride < (size_t)c->P * (c->P + 1)) return fail(c, SFMM_INVALID_ARG, "stride smaller than P(P+1)");
    cudaSetDevice(c->device);
    cudaError_t e = launch_p2x(c->dtype == SFMM_F64, kind, c->P, (long long)nexp, 0, offset, charge, pos, centre,
                               out, (long long)out_stride, c->num_sms, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "P2M/P2L kernel");
    c->launches++;
    return SFMM_OK;
}

int sfmm_eval_device(sfmm_context *c, int kind, size_t npts, const double *pos, const uint32_t *box,
                     const void *E, size_t stride, size_t nexp, const double *centre, double *potential,
                     double *gradient)
{
    if (!c) return SFMM_INVALID_ARG;
    Range range("sfmm l2p/m2p");
    if (kind != 0 && kind != 1) return fail(c, SFMM_INVALID_ARG, "kind must be 0 (L2P) or 1 (M2P)");
    if (npts == 0) return SFMM_OK;
    if (!pos || !E || !centre || !potential) return fail(c, SFMM_INVALID_ARG, "null device pointer");
    if (stride < (size_t)c->P * (c->P + 1)) return fail(c, SFMM_INVALID_ARG, "stride smaller than P(P+1)");
    if (gradient && kind != 0) return fail(c, SFMM_UNSUPPORTED, "gradients are evaluated for local expansions");
    if (!box && nexp < npts) return fail(c, SFMM_INVALID_ARG, "fewer expansions than points without a box index");
    cudaSetDevice(c->device);
    // float-float normalises all nexp expansions into scratch first: worth it
    // from one point per four expansions on.  The scratch is allocated (or
    // grown) outside stream capture only; a call without enough of it (in a
    // capture, or when the allocation fails) does without the gradient's
    // pairings, or runs the FP64 kernel.
    std::lock_guard<std::mutex> lk(c->eval_mtx);  // calls share the scratch, in stream order
    void *scratch = nullptr;
    bool pairings = false;
    const size_t need = 4 * npts >= nexp ? eval_scratch_bytes(c->P, (long long)nexp, false) : 0;
    if (need) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(c->stream, &cs);
        const bool capturing = cs != cudaStreamCaptureStatusNone;
        if (gradient && eval_wants_pairings(c->P, (long long)npts, (long long)nexp, c->num_sms)) {  // a buffer of its own: plain calls alone need a quarter of it
            scratch = c->d_eval_grad.take(eval_scratch_bytes(c->P, (long long)nexp, true), capturing);
            pairings = scratch != nullptr;
        }
        // a gradient call's buffer serves plain calls too, recorded ones among
        // them, which would run FP64 without (P=12, 100 000 points: 290 us for 64)
        if (!scratch) scratch = (c->d_eval.fits(need) || !c->d_eval_grad.fits(need) ? c->d_eval : c->d_eval_grad).take(need, capturing);
    }
    cudaError_t e = launch_eval(c->dtype == SFMM_F64, kind, c->P, (long long)npts, pos, box, E, (long long)stride,
                                (long long)nexp, centre, potential, gradient, scratch, pairings, c->num_sms, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "L2P/M2P kernel");
    c->launches++;
    return SFMM_OK;
}

}  // extern "C"
