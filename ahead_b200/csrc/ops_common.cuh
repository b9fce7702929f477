// ops_common.cuh -- pieces shared by the operator translation units: width
// dispatch, error-vector plumbing and the column check used for every
// error-position vector that is a plain "decode and compare" over a column.
#pragma once

#include <type_traits>

#include "context.cuh"

namespace ahead {

// Dispatch a functor on the storage width of a column type.
template <class F>
inline int by_width(int w, F&& f) {
    switch (w) {
        case 1: return f(std::integral_constant<int, 1>());
        case 2: return f(std::integral_constant<int, 2>());
        case 4: return f(std::integral_constant<int, 4>());
        default: return f(std::integral_constant<int, 8>());
    }
}

// Same for AN-coded columns, whose codes are 2, 4 or 8 bytes wide.
template <class F>
inline int by_width_enc(int w, F&& f) {
    switch (w) {
        case 2: return f(std::integral_constant<int, 2>());
        case 4: return f(std::integral_constant<int, 4>());
        default: return f(std::integral_constant<int, 8>());
    }
}


inline uint32_t grid_for(uint64_t n, int threads) {
    uint64_t g = (n + threads - 1) / threads;
    return (uint32_t)(g < 148 * 16 ? (g ? g : 1) : 148 * 16);
}

inline uint64_t ecap(const ahead_errvec* e) { return (e && e->data) ? e->capacity : 0; }
inline uint64_t* edata(const ahead_errvec* e) { return e ? e->data : nullptr; }


// checkAN: encdecAN_scalar.tcc:84-90.
template <int WW>
struct CheckOp {
    static constexpr int W = WW;
    static constexpr int NCH = 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = false;
    const char* base;
    uint32_t* status;
    uint64_t ainv, umax, aoid, errcap;
    uint64_t* err;
    uint64_t* acc;
    static constexpr bool EMIT_V = false;
    static constexpr int NOUT = 1;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t, uint64_t&) const {
        return mulw(v, ainv, W) > umax ? 1u : 0u;
    }
    AHEAD_DEV uint64_t out0(int, uint64_t, uint64_t row) const { return row * aoid; }
    AHEAD_DEV uint64_t cap0() const { return errcap; }
    AHEAD_DEV void* optr(int) const { return err; }
    AHEAD_DEV int owidth(int) const { return 8; }
    AHEAD_DEV void emit(int, uint64_t pos, uint64_t, uint64_t row) const {
        if (pos < errcap) err[pos] = row * aoid;
    }
};


// Error positions of one column: rows whose code, multiplied by ainv in the
// `wenc`-byte ring, exceeds umax (the check every AN operator applies to each
// of its encoded inputs, e.g. hashjoinAN.tcc:144-149).  Rows [0, n).
template <int WW>
struct ColCheckOp {
    static constexpr int W = WW;
    static constexpr int NCH = 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = false;
    static constexpr bool EMIT_V = false;
    static constexpr int NOUT = 1;
    const char* base;
    uint32_t* status;
    uint64_t ainv, umax, aoid, errcap, wmaskenc;
    uint64_t* err;
    uint64_t* acc;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t, uint64_t&) const { return ((v * ainv) & wmaskenc) > umax ? 1u : 0u; }
    AHEAD_DEV uint64_t out0(int, uint64_t, uint64_t row) const { return row * aoid; }
    AHEAD_DEV uint64_t cap0() const { return errcap; }
    AHEAD_DEV void* optr(int) const { return err; }
    AHEAD_DEV int owidth(int) const { return 8; }
    AHEAD_DEV void emit(int, uint64_t pos, uint64_t, uint64_t row) const {
        if (pos < errcap) err[pos] = row * aoid;
    }
};

inline size_t colcheck_scratch(uint64_t n) { return compact_scratch<ColCheckOp<8>>(n); }

// Launch the column check; the error count lands in counter `ci`.
inline void run_colcheck(OpScope& s, const ahead_col& c, uint64_t n, uint64_t ainv, uint64_t umax, int wenc,
                         uint64_t aoid, ahead_errvec* e, int ci) {
    if (!n || !e) return;
    by_width_enc(type_width(c.type), [&](auto tag) -> int {
        constexpr int W = decltype(tag)::value;
        ColCheckOp<W> op;
        op.base = (const char*)c.data;
        op.status = s.d_status;
        op.ainv = ainv;
        op.umax = umax;
        op.aoid = aoid;
        op.errcap = ecap(e);
        op.err = edata(e);
        op.wmaskenc = wmask(wenc);
        op.acc = nullptr;
        run_compact(s, op, n, ci);
        return 0;
    });
}

// ------------------------------------------------------- rare error rows
// Corrupt codes are rare, so the kernels that read a column anyway append the
// rows of corrupt codes to a short list (in any order); only when a list is
// not empty is it sorted into the error vector, and only when it overflows is
// the vector made by a compaction of the column.
constexpr uint32_t kFastErrCap = 4096;

// Block c sorts list c (at most kFastErrCap rows, bitonic in shared memory)
// and writes row * aoid into the error vector, up to its capacity; block 0
// also writes its sorted rows to `sorted` when given.
static __global__ void __launch_bounds__(1024) sort_err_rows_kernel(const unsigned long long* cnt, const uint64_t* rows1,
                                                             const uint64_t* rows2, uint64_t* e1, uint64_t cap1,
                                                             uint64_t* e2, uint64_t cap2, uint64_t aoid,
                                                             uint64_t* sorted = nullptr) {
    __shared__ uint64_t s_r[kFastErrCap];
    const int c = blockIdx.x;
    const unsigned long long k = cnt[c];
    uint64_t* e = c == 0 ? e1 : e2;
    const uint64_t cap = c == 0 ? cap1 : cap2;
    if (k == 0 || k > kFastErrCap) return;
    const uint64_t* rows = c == 0 ? rows1 : rows2;
    uint32_t m = 1;
    while (m < k) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) s_r[i] = i < k ? rows[i] : ~0ull;
    __syncthreads();
    for (uint32_t size = 2; size <= m; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                const uint32_t j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0;
                    const uint64_t x = s_r[i], y = s_r[j];
                    if ((x > y) == up) {
                        s_r[i] = y;
                        s_r[j] = x;
                    }
                }
            }
            __syncthreads();
        }
    if (e)
        for (uint32_t i = threadIdx.x; i < k && i < cap; i += blockDim.x) e[i] = s_r[i] * aoid;
    if (sorted && c == 0)
        for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) sorted[i] = s_r[i];
}

// One column's short error list: its count is counter `ci` of the call.
struct ErrList {
    unsigned long long* cnt;
    uint64_t* rows;  // [kFastErrCap]
    AHEAD_DEV void add(uint64_t row) const {
        if (*(volatile unsigned long long*)cnt > kFastErrCap) return;  // (a column of errors: no queue on one word)
        const unsigned long long k = atomicAdd(cnt, 1ull);
        if (k < kFastErrCap) rows[k] = row;
    }
};
constexpr size_t kErrListBytes = kFastErrCap * 8 + 256;

inline ErrList err_list(OpScope& s, int ci) {
    ErrList l;
    l.cnt = (unsigned long long*)(s.d_counters + ci);
    l.rows = (uint64_t*)s.alloc(kFastErrCap * 8);
    return l;
}

// After finish() has read the counters back: writes the error vector of a list
// with a few rows (a launch, no wait: the stream orders it before any reader)
// and returns false when the list overflowed, so that the caller runs the
// column's compaction.
inline bool settle_err_list(OpScope& s, const ErrList& l, int ci, uint64_t aoid, ahead_errvec* e) {
    const uint64_t k = s.counter(ci);
    if (k > kFastErrCap) return false;
    if (e) {
        e->count = k;
        if (k && edata(e)) {
            sort_err_rows_kernel<<<1, 1024, 0, s.ctx->stream>>>(l.cnt, l.rows, nullptr, edata(e), ecap(e), nullptr, 0,
                                                                aoid);
            s.launched();
        }
    }
    return true;
}

}  // namespace ahead

namespace ahead {
// ANhelper<V>::mulIfEncoded(x, f) on the host with f = the column's A^-1:
// (storage)(x * A^-1) for an encoded column, (storage)x otherwise.  Used for
// re-encoding factors A_new * A_old^-1 (hashjoinAN.tcc:95-96, matchjoinAN.tcc:80-81).
inline uint64_t dec_if_host(const DCol& c, uint64_t x) { return c.enc ? mulw(x, c.ainv, c.width) : (x & wmask(c.width)); }
}  // namespace ahead
