// Context internals shared by the C ABI (sfmm_capi.cpp) and the execution
// plans (sfmm_plan.cpp).  Not part of the public interface.
#pragma once

#include "sfmm.h"

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <atomic>
#include <cstdint>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <tuple>
#include <string>
#include <utility>
#include <vector>

#include "sfmm_hostbatch.hpp"
#include "sfmm_launch.hpp"
#include "sfmm_tables.hpp"

namespace sfmm {

// device tables of the FP64 kernel for orders above 32
struct DevTables {
    void *W = nullptr, *ein_M = nullptr, *ein_L = nullptr, *eout_L = nullptr, *eout_M = nullptr;
    void *H[3] = {nullptr, nullptr, nullptr};
    bool ready = false;
};

// Device tables of the 60-bit fixed-point, the FP32 or the split kernel
// (sfmm_tables.hpp, FxTables, F32Tables, SplitTables) in one allocation: a set
// per group size and the edge factors (e_in_M, e_in_L, e_out_L, e_out_M).
struct FxDevTables {
    const void *W = nullptr, *H[3] = {nullptr, nullptr, nullptr};
    int P = 0;
    std::vector<int> wend;  // bytes of the swap tables of degrees below an order bound
    int hbytes = 0;         // of one operator's z matrices
};
struct ArithTables {
    void *mem = nullptr;
    const void *edge[4] = {};
    FxDevTables group[2];  // 4 and 8 threads per translation
};

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t b)
    {
        if (b <= bytes) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, b);
        if (e == cudaSuccess) bytes = b;
        return e;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
};

// Scratch that calls recorded in a stream capture may point to: a buffer such
// a call took stays allocated until the context goes, since its graph may be
// replayed after the scratch has grown.
struct GraphBuf {
    DevBuf buf;
    bool recorded = false;
    std::vector<void *> kept;
    bool fits(size_t b) const { return b <= buf.bytes; }
    // b bytes, allocated or grown outside captures only; nullptr without them
    void *take(size_t b, bool capturing)
    {
        if (!fits(b)) {
            if (capturing) return nullptr;
            if (recorded) {
                try {
                    kept.push_back(buf.p);
                } catch (const std::bad_alloc &) {
                    return nullptr;
                }
                buf = DevBuf{};
                recorded = false;
            }
            if (buf.ensure(b) != cudaSuccess) {
                (void)cudaGetLastError();
                return nullptr;
            }
        }
        recorded = recorded || capturing;
        return buf.p;
    }
    void release()
    {
        buf.release();
        for (void *p : kept) cudaFree(p);
        kept.clear();
    }
};

struct HostBuf {
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t b)
    {
        if (b <= bytes) return cudaSuccess;
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMallocHost(&p, b);
        if (e == cudaSuccess) bytes = b;
        return e;
    }
    void release()
    {
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
    }
};

}  // namespace sfmm

struct sfmm_context {
    int dtype = SFMM_F64;
    int P = 0;
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    sfmm::HostTables host;
    sfmm::DevTables tab;  // FP64 above order 32
    sfmm::ArithTables fxt[sfmm::kNumArith];  // by Arith
    sfmm::TcDevTables *tc[3] = {nullptr, nullptr, nullptr};  // tensor-core operand images by format
    std::string err;
    std::atomic<uint64_t> launches{0};
    std::mutex mtx;  // serialises host-path calls (one translator object, one stream)
    std::mutex setup_mtx;  // table uploads and the launch-shape cache (device calls may come from several threads)
    std::mutex eval_mtx;   // the L2P/M2P scratch (d_eval, d_eval_grad): sized and used by one call at a time
    int *d_status = nullptr;  // device error word of the translation kernels
    // host-path staging (three pipeline slots for the packed host call)
    sfmm::DevBuf d_src[3], d_dst[3], d_meta[3], d_shift[3], d_work;
    sfmm::GraphBuf d_eval;       // normalised expansions of the float-float L2P/M2P
    sfmm::GraphBuf d_eval_grad;  // the same with the gradient's pairings
    sfmm::HostBuf h_src, h_dst, h_meta, h_shift;
    cudaStream_t pipe[3] = {nullptr, nullptr, nullptr};
    // (op, mode, order bound) -> launch shape: operators tuned apart keep
    // their own shapes at one order
    std::map<std::tuple<int, int, int>, sfmm::LaunchShape> shapes;
    int *d_woff = nullptr, *d_hoff = nullptr;            // offsets of tab's blocks
    bool pageable_access = false;  // the GPU reads pageable host memory through the host page tables
    sfmm::SlotScratch slot_scratch;  // target table of the classic host call
    std::set<std::tuple<int, int, int>> tuned;  // (op, mode, order bound) shapes measured by sfmm_tune
};

namespace sfmm {

// NVTX range over a scope, shown by profilers on the host timeline (a no-op
// unless a tool is attached)
struct Range {
    explicit Range(const char *name) { nvtxRangePushA(name); }
    ~Range() { nvtxRangePop(); }
    Range(const Range &) = delete;
    Range &operator=(const Range &) = delete;
};

// record an error on the context and return the status
int fail(sfmm_context *c, int st, const char *fmt, ...);
int cuda_fail(sfmm_context *c, cudaError_t e, const char *what);
// arithmetic of a precision mode on this context
int arith_of(sfmm_context *c, int precision, Arith *out);
// upload the arithmetic's tables once (setup_mtx held)
int ensure_tables(sfmm_context *c, Arith a);
// The mode a batch of op with this order bound runs in (split M2M above order
// 18 runs as split_ff, tensor-core modes above order 16 as split): launch
// shapes, pinned or measured, belong to it.
Arith resolve_mode(Arith a, int op, int Pbound);
// the arithmetic of that mode's kernel (split_ff runs plain FP64's)
Arith resolve_arith(Arith a, int op, int Pbound);
// device address of a caller's host array when the kernels can use it
// directly (pinned host memory, or pageable memory on a GPU that uses the host
// page tables), else nullptr
const void *device_view(sfmm_context *c, const void *host);
// tables and launch shape of (arithmetic, order bound) for op, so that a
// launch makes no allocation (plans call this before a graph capture)
int prepare_launch(sfmm_context *c, int op, Arith a, int Pbound, LaunchShape *shape = nullptr);
// replace (or, with nullptr, drop) the cached launch shape of (op, mode, order bound)
void set_shape(sfmm_context *c, std::tuple<int, int, int> key, const LaunchShape *s);
// one validated translation launch on device pointers (translation i of the
// batch is perm[i] when perm is given)
// A work list (work, work_counter, nwork: see KParams) turns the launch into
// one persistent grid that takes its tiles from the list; `shape` (may be
// null) replaces the context's launch shape for this launch.
struct WorkList {
    const uint2 *work = nullptr;
    unsigned *counter = nullptr;
    long long n = 0;
};
int run_batch(sfmm_context *c, cudaStream_t stream, int op, Arith a, int Pbound, long long n, const void *src,
              long long sstride, long long nsrc, const uint32_t *sidx, void *dst, long long dstride, long long ndst,
              const uint32_t *tidx, const uint32_t *pin, const uint32_t *pout, const double *shift,
              const uint32_t *perm, int flags, long long nidx = -1,
              const unsigned long long *src_ptr = nullptr, const unsigned long long *dst_ptr = nullptr,
              bool in_hbm = true, const WorkList *wl = nullptr, const LaunchShape *shape = nullptr);

}  // namespace sfmm
