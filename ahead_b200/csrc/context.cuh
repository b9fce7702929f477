// context.cuh -- the ahead_ctx behind the C ABI and the per-call scope that
// carves device scratch out of the context's arena.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <memory>
#include <string>

#include "../../include/ahead_gpu.h"
#include "common.cuh"
#include "compact.cuh"

struct ahead_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    char* arena = nullptr;  // device scratch, reused by every call
    size_t arena_cap = 0;
    bool header_clean = false;  // the arena's counters are zero
    uint64_t* h_stage = nullptr;  // pinned host words for count read-back (device-writable)
    uint64_t launches = 0;
    int num_sms = 148;
    std::string err;
    ahead_output_fn out_fn = nullptr;  // allocates output columns of sized calls
    void* out_user = nullptr;
    // staging buffers of the table loader (pinned host + device text blocks),
    // kept across loads; freed with the context
    std::shared_ptr<void> loader;
};

namespace ahead {

constexpr int kStageWords = 64;
constexpr int kScanDone = 61;  // counter word of tile_scan_kernel

// noalloc.cu: drop the cached scratch address of a device (a new context may
// follow a device reset).
void noalloc_forget_device(int dev);

inline int fail(ahead_ctx* ctx, int status, const std::string& what) {
    if (ctx) ctx->err = what;
    return status;
}

inline int cuda_fail(ahead_ctx* ctx, cudaError_t e, const char* where) {
    return fail(ctx, AHEAD_CUDA_ERROR, std::string(where) + ": " + cudaGetErrorString(e));
}

#define AHEAD_CUDA(ctx, call)                                      \
    do {                                                           \
        cudaError_t _e = (call);                                   \
        if (_e != cudaSuccess) return ::ahead::cuda_fail((ctx), _e, #call); \
    } while (0)

// Ends an operator: the first `n` counters (words 1 to n) go to the pinned host
// words, and the header is left zero for the next call.  (A copy to the
// host and a clear ahead of the next call's kernels cost each call 7 us more.)
static __global__ void __launch_bounds__(kStageWords) publish_kernel(uint64_t* header, uint64_t* host, int n) {
    const int i = threadIdx.x;
    const uint64_t v = header[i];
    if (i <= n) host[i] = v;
    if (v) header[i] = 0;
}

// One operator call.  Layout of the arena: [a spare word, 63 counters][bump
// region].  reserve() must be called with the call's total scratch need
// before any pointer is handed out (it may reallocate the arena).
struct OpScope {
    ahead_ctx* ctx;
    size_t off = 0;
    uint64_t* d_counters = nullptr;  // [kStageWords - 1]
    int rc = AHEAD_OK;
    bool pending = false;  // launches since the last wait

    explicit OpScope(ahead_ctx* c) : ctx(c) {}

    int reserve(size_t bytes) {
        size_t need = 512 + bytes + 256;
        if (need > ctx->arena_cap) {
            cudaError_t e = cudaStreamSynchronize(ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaStreamSynchronize");
            if (ctx->arena) cudaFree(ctx->arena);
            ctx->arena = nullptr;
            ctx->header_clean = false;
            size_t cap = need < (64u << 20) ? (64u << 20) : need + need / 4;
            e = cudaMalloc(&ctx->arena, cap);
            if (e != cudaSuccess) {
                cudaGetLastError();  // (not sticky: the caller may do with less)
                ctx->arena_cap = 0;
                return fail(ctx, AHEAD_NO_MEMORY, "scratch arena allocation failed");
            }
            ctx->arena_cap = cap;
        }
        d_counters = (uint64_t*)(ctx->arena + 8);
        off = 512;
        if (!ctx->header_clean) {
            cudaError_t e = cudaMemsetAsync(ctx->arena, 0, 512, ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMemsetAsync");
        }
        ctx->header_clean = false;  // (until finish() has run: a call may fail half way)
        return AHEAD_OK;
    }

    void* alloc(size_t bytes) {
        off = (off + 255) & ~size_t(255);
        void* p = ctx->arena + off;
        off += bytes;
        return p;
    }

    // Compaction scratch for n rows in `ntiles` tiles and `nchan` streams; the stream
    // totals land in d_counters[first_counter ...].  Every word is written
    // before it is read; the scan's `done` word leaves each scan as zero.
    CompactBufs compact_bufs(uint64_t n, uint32_t ntiles, uint32_t nchan, int first_counter) {
        CompactBufs cb;
        cb.words = (uint32_t*)alloc((size_t)(n + 1023) / 1024 * 128);
        cb.counts = (uint32_t*)alloc((size_t)ntiles * nchan * 4);
        cb.offsets = (uint64_t*)alloc((size_t)ntiles * nchan * 8);
        cb.gbase = (uint64_t*)alloc((size_t)scan_groups(ntiles) * nchan * 8);
        cb.totals = d_counters + first_counter;
        cb.done = (uint32_t*)(d_counters + kScanDone);
        cb.ntiles = ntiles;
        cb.nchan = nchan;
        return cb;
    }

    void launched(int n = 1) {
        ctx->launches += n;
        pending = true;
        ctx->header_clean = false;
    }

    // Waits for launches made after the last finish(): a caller may read the
    // outputs on any stream once a call has returned.
    int wait() {
        if (!pending) return AHEAD_OK;
        pending = false;
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(ctx, e, "kernel launch");
        e = cudaStreamSynchronize(ctx->stream);
        return e == cudaSuccess ? AHEAD_OK : cuda_fail(ctx, e, "cudaStreamSynchronize");
    }

    // Read the first `ncounters` counters back and wait for the stream.  The
    // device's counters are zero from here on.
    int finish(int ncounters) {
        pending = false;
        publish_kernel<<<1, kStageWords, 0, ctx->stream>>>((uint64_t*)ctx->arena, ctx->h_stage, ncounters);
        ctx->launches += 1;
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(ctx, e, "kernel launch");
        e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaStreamSynchronize");
        ctx->header_clean = true;
        return AHEAD_OK;
    }
    uint64_t counter(int i) const { return ctx->h_stage[1 + i]; }

    // A call whose output columns are allocated once its counts are known.
    bool sized(const ahead_bat* out, uint64_t cap) const {
        return ctx->out_fn && cap == AHEAD_SIZED && !out->head.data && !out->tail.data;
    }
    // The column's buffer of `rows` rows; false when the caller's function has none.
    bool take(ahead_col* c, int column, uint64_t rows) {
        c->data = ctx->out_fn(ctx->out_user, column, (rows ? rows : 1) * (uint64_t)type_width(c->type));
        return c->data != nullptr;
    }
    // An output without rows: a sized call still gets its columns.
    int empty(ahead_bat* out, uint64_t cap, bool tail) {
        if (sized(out, cap) && (!take(&out->head, 0, 0) || (tail && !take(&out->tail, 1, 0))))
            return fail(ctx, AHEAD_NO_MEMORY, "output allocation failed");
        return AHEAD_OK;
    }
};

inline DCol dcol(const ahead_col& c) {
    DCol d;
    d.data = c.data;
    d.seqbase = c.seqbase;
    d.type = c.type;
    d.width = type_width(c.type);
    d.enc = type_encoded(c.type);
    d.ainv = d.enc ? (c.Ainv & wmask(d.width)) : 0;
    d.umax = c.unenc_max & wmask(d.width);
    d.pad = 0;
    return d;
}

inline void set_meta(ahead_col* c, int type, uint64_t A, uint64_t Ainv, uint64_t umax, uint64_t seq) {
    c->type = type;
    c->A = (uint16_t)A;  // ColumnMetaData::AN_A is a 16-bit A_t
    c->Ainv = Ainv;
    c->unenc_max = umax;
    c->seqbase = seq;
}
inline void copy_meta(ahead_col* c, int type, const ahead_col* src) {
    set_meta(c, type, src->A, src->Ainv, src->unenc_max, src->seqbase);
}
// ColumnDescriptor's default metadata: A=1, Ainv=1, unencMaxU=0 and, for a
// non-void column, seqbase = sizeof(type_t) (ColumnDescriptor.hpp:39-41 picks
// the oid_t seqbase constructor of ColumnMetaData).
inline void default_meta(ahead_col* c, int type) {
    set_meta(c, type, 1, 1, 0, type == AHEAD_VOID ? 0 : (uint64_t)type_width(type));
}
inline uint64_t type_unenc_max(int t) {
    switch (t) {
        case AHEAD_RESTINY: return 0xFF;
        case AHEAD_RESSHORT: return 0xFFFF;
        case AHEAD_RESINT: return 0xFFFFFFFFull;
        default: return kRes56Max;
    }
}

inline void ev_begin(ahead_errvec* e, int present) {
    if (!e) return;
    e->present = present;
    e->count = 0;
}

// Modular inverse of odd a modulo 2^bits (Newton iteration x <- x(2 - ax)).
inline uint64_t inv_pow2(uint64_t a, int bits) {
    uint64_t x = a;  // correct to 3 bits for odd a
    for (int i = 0; i < 6; ++i) x *= 2 - a * x;
    return x & wmask(bits / 8);
}

// A kernel's dynamic shared-memory limit is a function attribute of each
// device: set it once per device (the context's, current in the calling
// thread), tracked per kernel in a set of devices 0..63 (beyond that it is
// set on every call).  False when the attribute could not be set.
template <auto Kernel>
inline bool dyn_smem_ready(const ahead_ctx* ctx, int bytes) {
    static std::atomic<uint64_t> done{0};
    const int dev = ctx->device;
    const uint64_t bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return true;
    if (cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        cudaGetLastError();  // (not sticky)
        return false;
    }
    if (bit) done.fetch_or(bit, std::memory_order_acq_rel);
    return true;
}

inline uint32_t tiles_per_warp(const ahead_ctx* ctx, uint32_t nt) {
    const uint32_t k = nt / ((uint32_t)ctx->num_sms * 8 * kCWarps);
    return k < 1 ? 1 : k > 8 ? 8 : k;
}

// Launch one compaction over n rows with its scratch in `cb`; returns the
// number of launches.  Few tiles: one block does everything (the separate
// launches of almost no work each cost 15 us at 2,556 rows, the one 5).  Else 1
// to 8 tiles per warp, so that the grid keeps about eight blocks per SM busy.
template <class Op>
inline int launch_compact(const ahead_ctx* ctx, cudaStream_t st, const Op& op, uint64_t n, const CompactBufs& cb) {
    const uint32_t nt = cb.ntiles;
    if (nt <= kOneBlockTiles && !long_tiles<Op>(n)) {
        compact_one_kernel<Op><<<1, nt * 32, 0, st>>>(op, n, cb);
        return 1;
    }
    const uint32_t per = tiles_per_warp(ctx, nt);
    const uint32_t grid = (nt + per * kCWarps - 1) / (per * kCWarps);
    auto passes = [&](auto k_tag) {
        constexpr int K = decltype(k_tag)::value;
        classify_kernel<Op, K><<<grid, kCThreads, 0, st>>>(op, n, cb, (int)per);
        const int scans = scan_tiles(st, cb);
        emit_kernel<Op, K><<<grid, kCThreads, 0, st>>>(op, n, cb, (int)per);
        return 2 + scans;
    };
    if constexpr (!Op::GATHER)
        if (long_tiles<Op>(n)) return passes(std::integral_constant<int, kLongK>());
    return passes(std::integral_constant<int, short_k(Op::W)>());
}

// The compaction of a sized call: counts first, then `alloc(kept)` sets the op's
// output pointers and capacity, then the rows.  Reads `ncounters` counters back.
template <class Op, class Alloc>
inline int run_compact_sized(OpScope& s, Op& op, uint64_t n, int c0, int ncounters, Alloc&& alloc) {
    const uint32_t nt = compact_tiles<Op>(n), per = tiles_per_warp(s.ctx, nt);
    const CompactBufs cb = s.compact_bufs(n, nt, Op::NCH, c0);
    const uint32_t grid = (nt + per * kCWarps - 1) / (per * kCWarps);
    cudaStream_t st = s.ctx->stream;
    auto passes = [&](auto k_tag) -> int {
        constexpr int K = decltype(k_tag)::value;
        classify_kernel<Op, K><<<grid, kCThreads, 0, st>>>(op, n, cb, (int)per);
        s.launched(1 + scan_tiles(st, cb));
        int rc = s.finish(ncounters);
        if (rc) return rc;
        if (!alloc(s.counter(c0))) return fail(s.ctx, AHEAD_NO_MEMORY, "output allocation failed");
        emit_kernel<Op, K><<<grid, kCThreads, 0, st>>>(op, n, cb, (int)per);
        s.launched();
        return s.wait();
    };
    if constexpr (!Op::GATHER)
        if (long_tiles<Op>(n)) return passes(std::integral_constant<int, kLongK>());
    return passes(std::integral_constant<int, short_k(Op::W)>());
}

// Passes 2 and 3 of a compaction in short tiles whose pass 1 has its own kernel.
template <class Op>
inline void launch_emit(OpScope& s, const Op& op, uint64_t n, const CompactBufs& cb) {
    constexpr int K = short_k(Op::W);
    const uint32_t per = tiles_per_warp(s.ctx, cb.ntiles);
    emit_kernel<Op, K><<<(cb.ntiles + per * kCWarps - 1) / (per * kCWarps), kCThreads, 0, s.ctx->stream>>>(op, n, cb,
                                                                                                           (int)per);
    s.launched();
}
inline void launch_scan(OpScope& s, const CompactBufs& cb) {
    s.launched(scan_tiles(s.ctx->stream, cb));
}

// A compaction of an operator call; totals land in counters [c0, c0 + NCH).
template <class Op>
inline void run_compact(OpScope& s, const Op& op, uint64_t n, int c0) {
    if (n == 0) return;
    const CompactBufs cb = s.compact_bufs(n, compact_tiles<Op>(n), Op::NCH, c0);
    s.launched(launch_compact(s.ctx, s.ctx->stream, op, n, cb));
}

template <class Op>
inline size_t compact_scratch(uint64_t n) {
    if (n == 0) return 0;
    return compact_bytes(n, compact_tiles<Op>(n), Op::NCH) + 1024;
}

}  // namespace ahead
