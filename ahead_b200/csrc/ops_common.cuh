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
    uint64_t ainv, umax, aoid, errcap, wmaskenc;
    uint64_t* err;
    uint64_t* acc;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t, uint64_t&) const { return ((v * ainv) & wmaskenc) > umax ? 1u : 0u; }
    AHEAD_DEV uint64_t out0(int, uint64_t, uint64_t row) const { return row * aoid; }
    AHEAD_DEV uint64_t cap0() const { return errcap; }
    AHEAD_DEV void* optr(int) const { return err; }
    AHEAD_DEV int owidth(int) const { return 8; }
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

// Sorts m words of shared memory (a power of two), by the whole block: bitonic, the
// steps between words less than 32 apart in registers, so that a barrier follows
// only 40 of 4,096 words' 78 steps.
AHEAD_DEV void sort_block(uint64_t* s, uint32_t m) {
    for (uint32_t size = 2; size <= m; size <<= 1) {
        uint32_t stride = size >> 1;
        for (; stride >= 32; stride >>= 1) {
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                const uint32_t j = i ^ stride;
                if (j > i) {
                    const uint64_t x = s[i], y = s[j];
                    if ((x > y) == ((i & size) == 0)) {
                        s[i] = y;
                        s[j] = x;
                    }
                }
            }
            __syncthreads();
        }
        for (uint32_t i = threadIdx.x; (i & ~31u) < m; i += blockDim.x) {  // (whole warps)
            uint64_t x = i < m ? s[i] : ~0ull;
            for (uint32_t d = stride; d > 0; d >>= 1) {
                const uint64_t y = __shfl_xor_sync(kFull, x, d);
                const bool low = ((i & d) == 0) == ((i & size) == 0);  // keeps the smaller of the two
                if ((y < x) == low) x = y;
            }
            if (i < m) s[i] = x;
        }
        __syncthreads();
    }
}

// Block c sorts list c (at most kFastErrCap rows, bitonic in shared memory)
// and writes row * aoid into the error vector, up to its capacity.  The counts
// come from the device (`cnt`), or for one list from the host (`known`).
static __global__ void __launch_bounds__(1024) sort_err_rows_kernel(const unsigned long long* cnt, uint64_t known,
                                                             const uint64_t* rows1, const uint64_t* rows2, uint64_t* e1,
                                                             uint64_t cap1, uint64_t* e2, uint64_t cap2,
                                                             uint64_t aoid) {
    __shared__ uint64_t s_r[kFastErrCap];
    const int c = blockIdx.x;
    const unsigned long long k = cnt ? cnt[c] : known;
    uint64_t* e = c == 0 ? e1 : e2;
    const uint64_t cap = c == 0 ? cap1 : cap2;
    if (k == 0 || k > kFastErrCap) return;
    const uint64_t* rows = c == 0 ? rows1 : rows2;
    uint32_t m = 1;
    while (m < k) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) s_r[i] = i < k ? rows[i] : ~0ull;
    __syncthreads();
    sort_block(s_r, m);
    if (e)
        for (uint32_t i = threadIdx.x; i < k && i < cap; i += blockDim.x) e[i] = s_r[i] * aoid;
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
// with a few rows (a launch: the caller waits) and returns false when the list
// overflowed, so that the caller runs the column's compaction.
inline bool settle_err_list(OpScope& s, const ErrList& l, int ci, uint64_t aoid, ahead_errvec* e) {
    const uint64_t k = s.counter(ci);
    if (k > kFastErrCap) return false;
    if (e) {
        e->count = k;
        if (k && edata(e)) {
            sort_err_rows_kernel<<<1, 1024, 0, s.ctx->stream>>>(nullptr, k, l.rows, nullptr, edata(e), ecap(e),
                                                                nullptr, 0, aoid);
            s.launched();
        }
    }
    return true;
}

// Rows 2p and 2p + 1 of a column in one load (`vec`: its data is aligned to two rows).
template <int W>
AHEAD_DEV void load_pair(const char* data, uint64_t p, bool vec, uint64_t (&x)[2]) {
    if (vec) {
        if constexpr (W == 8) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(data) + p);
            x[0] = (uint64_t)q.y << 32 | q.x;
            x[1] = (uint64_t)q.w << 32 | q.z;
        } else if constexpr (W == 4) {
            const uint2 q = __ldg(reinterpret_cast<const uint2*>(data) + p);
            x[0] = q.x;
            x[1] = q.y;
        } else {
            static_assert(W == 2, "two-, four- and eight-byte columns");
            const uint32_t q = __ldg(reinterpret_cast<const uint32_t*>(data) + p);
            x[0] = q & 0xffffu;
            x[1] = q >> 16;
        }
    } else {
        x[0] = gmem_ld<W>(data, 2 * p);
        x[1] = gmem_ld<W>(data, 2 * p + 1);
    }
}
inline bool pair_aligned(const void* p, int w) { return (uintptr_t)p % (2 * w) == 0; }

// ---------------------------------------------- rows dropped now and then
// checkAndDecodeAN and the positional joins drop a row only when its code, OID
// or fetched value is corrupt, which is rare.  So one pass writes every row's
// output at the row's own position and lists the rows to drop (unordered; bit 0
// of an entry is its kind, which error vector reports it).  With none listed
// the outputs are done; with a few, the list is sorted into the error vectors
// and the outputs are moved down in place; more than kMaxDrops (or than the scratch
// holds the edges of): the caller
// runs the compaction, which writes everything again.  (The compaction's two
// passes gather every value twice.)
constexpr uint32_t kMaxDrops = 2048;
constexpr uint32_t kSureDrops = 256;  // scratch for the edges of this many is always there: an eighth of the outputs

struct DropList {
    unsigned long long *cnt, *kind1;  // entries, and those of kind 1
    uint64_t* rows;                   // [kMaxDrops] row << 1 | kind
    // true: more than kMaxDrops rows are dropped, so the caller's pass is for nothing
    AHEAD_DEV bool add(uint64_t row, uint32_t kind) const {
        if (*(volatile unsigned long long*)cnt > kMaxDrops) return true;
        const unsigned long long k = atomicAdd(cnt, 1ull);
        if (k < kMaxDrops) rows[k] = row << 1 | kind;
        if (kind) atomicAdd(kind1, 1ull);
        return false;
    }
};

inline DropList drop_list(OpScope& s, int ci) {  // counters ci, ci + 1
    DropList l;
    l.cnt = (unsigned long long*)(s.d_counters + ci);
    l.kind1 = l.cnt + 1;
    l.rows = (uint64_t*)s.alloc(kMaxDrops * 8);
    return l;
}

// One block sorts the k listed rows into `sorted` and writes the error vectors:
// row * aoid (kind 0, and kind 1 without a position column), or the position the
// row's OID names, times aoid (kind 1; `oid` holds the 8-byte codes).
static __global__ void __launch_bounds__(1024) sort_drops_kernel(const uint64_t* rows, uint32_t k, uint64_t* sorted,
                                                                 const uint64_t* oid, uint64_t ainv, uint64_t aoid,
                                                                 uint64_t* e0, uint64_t cap0, uint64_t* e1,
                                                                 uint64_t cap1) {
    __shared__ uint64_t s_r[kMaxDrops];
    __shared__ uint64_t s_part[33];
    uint32_t m = 1;
    while (m < k) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) s_r[i] = i < k ? rows[i] : ~0ull;
    __syncthreads();
    sort_block(s_r, m);
    uint64_t ones = 0;  // entries of kind 1 before this round's
    for (uint32_t i0 = 0; i0 < k; i0 += 1024) {
        const uint32_t i = i0 + threadIdx.x;
        const uint64_t x = i < k ? s_r[i] : 0;
        uint64_t total;
        const uint64_t before = ones + block_scan_1024(x & 1, s_part, &total);
        if (i < k) {
            const uint64_t row = x >> 1;
            sorted[i] = row;
            if (x & 1) {
                if (e1 && before < cap1) e1[before] = (oid ? oid[row] * ainv : row) * aoid;
            } else if (e0 && i - before < cap0) {
                e0[i - before] = row * aoid;
            }
        }
        ones += total;
    }
}

// Moves the rows of one or two columns (4-byte aligned) down over the k dropped
// ones, in place.  A chunk of 16 KB moves by at most k of its rows: the rows
// whose place lies in their own chunk go there directly, once all of the chunk
// has been read; the few that go to the chunk before wait in `edge` (k per chunk)
// for shift_edges_kernel.  Together they read and write each row behind the first
// dropped one once.  A chunk's loads are issued before it looks for its place in
// the list, which the whole block does with one load per entry.  1- and 2-byte
// rows are read and written as words shifted to their place: 150M 2-byte values
// move in 76 us (600 MB; checkAndDecodeAN with 3 flips, from 459 us with a row at
// a time and a result copied to its size to 313).  60M 4-byte values move in 88 us
// (480 MB, 5.5 TB/s); with a binary search ahead of the loads, or the rows spilled
// to local memory, it took 106 and 141.
constexpr uint32_t kShiftChunk = 2048;
constexpr uint32_t shift_chunk(int w) { return kShiftChunk * (8 / w); }

template <int W>
struct UIntOf {
    typedef typename std::conditional<W == 8, uint64_t, typename std::conditional<W == 4, uint32_t,
        typename std::conditional<W == 2, uint16_t, uint8_t>::type>::type>::type type;
};

struct ShiftCols {
    void* data[2];
    void* edge[2];
    uint64_t n;
    const uint64_t* sorted;
    uint32_t k;
};

AHEAD_DEV uint32_t drops_below(const uint64_t* sorted, uint32_t lo, uint32_t hi, uint64_t row) {
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg((const unsigned long long*)sorted + mid) < row) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

template <int W>
__global__ void __launch_bounds__(256, 8) shift_rows_kernel(ShiftCols s) {
    typedef typename UIntOf<W>::type T;
    constexpr uint32_t C = shift_chunk(W);
    constexpr uint32_t U = C / 256;
    const int col = blockIdx.y;
    const uint64_t c0 = (uint64_t)blockIdx.x * C;
    T* p = (T*)(col ? s.data[1] : s.data[0]) + c0;
    const uint32_t m = s.n - c0 < C ? (uint32_t)(s.n - c0) : C, t = threadIdx.x;
    if constexpr (W < 4) {  // (by words: a row at a time is as many loads and stores of a quarter or half of the bytes)
        constexpr uint32_t P = 4 / W, UW = C / P / 256;
        __shared__ __align__(16) uint32_t s_w[C / P + 1];
        uint32_t x[UW];
#pragma unroll
        for (uint32_t u = 0; u < UW; ++u) {
            const uint32_t r = (u * 256 + t) * P;
            x[u] = 0;
            if (r + P <= m) {
                x[u] = reinterpret_cast<const uint32_t*>(p)[u * 256 + t];
            } else {
                for (uint32_t i = 0; r + i < m; ++i) x[u] |= (uint32_t)p[r + i] << (8 * W * i);
            }
        }
        uint32_t lo = 0, hi = 0;
        for (uint32_t i0 = 0; i0 < s.k; i0 += 256) {
            const uint64_t r = i0 + t < s.k ? __ldg((const unsigned long long*)s.sorted + i0 + t) : ~0ull;
            lo += __syncthreads_count(r < c0);
            hi += __syncthreads_count(r < c0 + m);
        }
        if (hi == 0) return;
#pragma unroll
        for (uint32_t u = 0; u < UW; ++u) s_w[u * 256 + t] = x[u];
        if (t == 0) s_w[C / P] = 0;
        __syncthreads();
        const T* s_r = reinterpret_cast<const T*>(s_w);
        T* e = (T*)(col ? s.edge[1] : s.edge[0]) + (uint64_t)blockIdx.x * s.k;
        if (lo == hi) {
            for (uint32_t r = t; r < lo && r < m; r += 256) e[lo - 1 - r] = s_r[r];
            const uint32_t left = m > lo ? m - lo : 0, by = lo % P;  // rows that stay in the chunk
            for (uint32_t j = t; j < left / P; j += 256) {
                const uint32_t at = j + lo / P;
                reinterpret_cast<uint32_t*>(p)[j] = __funnelshift_r(s_w[at], s_w[at + 1], 8 * W * by);
            }
            for (uint32_t r = (left / P) * P + t; r < left; r += 256) p[r] = s_r[lo + r];
            return;
        }
        for (uint32_t r = t; r < m; r += 256) {
            const uint32_t d = drops_below(s.sorted, lo, hi, c0 + r);
            if (d < hi && __ldg((const unsigned long long*)s.sorted + d) == c0 + r) continue;
            if (r >= d) p[r - d] = s_r[r];
            else e[d - 1 - r] = s_r[r];
        }
        return;
    }
    __shared__ T s_v[W < 4 ? 1 : C];
    typename std::conditional<W == 8, uint64_t, uint32_t>::type v[U];
    if (m == C) {
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) v[u] = p[u * 256 + t];
    } else {
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) v[u] = u * 256 + t < m ? p[u * 256 + t] : 0;
    }
    uint32_t lo = 0, hi = 0;  // dropped rows before the chunk, and before its end
    for (uint32_t i0 = 0; i0 < s.k; i0 += 256) {
        const uint64_t x = i0 + t < s.k ? __ldg((const unsigned long long*)s.sorted + i0 + t) : ~0ull;
        lo += __syncthreads_count(x < c0);  // (also: the chunk is read before any of it is overwritten)
        hi += __syncthreads_count(x < c0 + m);
    }
    if (hi == 0) return;
    T* e = (T*)(col ? s.edge[1] : s.edge[0]) + (uint64_t)blockIdx.x * s.k;
    if (lo == hi) {  // (nearly every chunk) the same move for all rows
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t r = u * 256 + t;
            if (r < lo) {
                if (r < m) e[lo - 1 - r] = (T)v[u];
            } else if (r < m) {
                p[r - lo] = (T)v[u];
            }
        }
        return;
    }
    // a chunk with dropped rows: each row looks up how many lie before it (through
    // shared memory: a loop of searches over a register array would spill it)
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) s_v[u * 256 + t] = (T)v[u];
    __syncthreads();
    for (uint32_t r = t; r < m; r += 256) {
        const uint32_t d = drops_below(s.sorted, lo, hi, c0 + r);
        if (d < hi && __ldg((const unsigned long long*)s.sorted + d) == c0 + r) continue;
        if (r >= d) p[r - d] = s_v[r];
        else e[d - 1 - r] = s_v[r];
    }
}

template <int W>
__global__ void __launch_bounds__(256) shift_edges_kernel(ShiftCols s) {  // a warp per chunk
    const int col = blockIdx.y;
    typedef typename UIntOf<W>::type T;
    constexpr uint32_t C = shift_chunk(W);
    const uint32_t lane = threadIdx.x & 31, chunk = blockIdx.x * 8 + (threadIdx.x >> 5);
    const uint64_t c0 = (uint64_t)chunk * C, c1 = c0 + C < s.n ? c0 + C : s.n;
    if (c0 >= s.n) return;
    uint32_t lo = 0, hi = 0;
    for (uint32_t i = lane; i < s.k; i += 32) {
        const uint64_t x = __ldg((const unsigned long long*)s.sorted + i);
        lo += x < c0;
        hi += x < c1;
    }
    lo = __reduce_add_sync(kFull, lo);
    hi = __reduce_add_sync(kFull, hi);
    const uint32_t clean = (uint32_t)(c1 - c0) - (hi - lo);
    const T* e = (const T*)(col ? s.edge[1] : s.edge[0]) + (uint64_t)chunk * s.k;
    T* p = (T*)(col ? s.data[1] : s.data[0]);
    // the chunk's first clean row goes to c0 - lo, the next ones behind it
    for (uint32_t i = lane; i < lo && i < clean; i += 32) p[c0 - lo + i] = e[lo - 1 - i];
}

// Scratch of the list, the sorted rows and the edges of columns of `row_bytes` together.
inline size_t drop_scratch(uint64_t n, uint64_t row_bytes) {
    return ((n + kShiftChunk - 1) / kShiftChunk) * kSureDrops * row_bytes + 2 * kMaxDrops * 8 + 4096;
}
// Whether k dropped rows' outputs (of `row_bytes` together) can be moved with the scratch at hand.
inline bool shift_fits(const OpScope& s, uint64_t n, uint64_t k, uint64_t row_bytes) {
    return k <= kMaxDrops &&
           s.off + ((n + kShiftChunk - 1) / kShiftChunk) * k * row_bytes + 1024 <= s.ctx->arena_cap;
}

// Closes the k gaps in the columns o and, when given, ot.
inline void launch_shift(OpScope& s, uint64_t n, const uint64_t* sorted, uint32_t k, void* o, int ow,
                         void* ot = nullptr, int otw = 0) {
    ShiftCols c;
    c.n = n;
    c.sorted = sorted;
    c.k = k;
    auto run = [&](int w, int cols) {
        by_width(w, [&](auto tag) -> int {
            constexpr int W = decltype(tag)::value;
            const uint32_t chunks = (uint32_t)((n + shift_chunk(W) - 1) / shift_chunk(W));
            for (int i = 0; i < cols; ++i) c.edge[i] = s.alloc((size_t)chunks * k * W);
            shift_rows_kernel<W><<<dim3(chunks, cols), 256, 0, s.ctx->stream>>>(c);
            shift_edges_kernel<W><<<dim3((chunks + 7) / 8, cols), 256, 0, s.ctx->stream>>>(c);
            return 0;
        });
        s.launched(2);
    };
    c.data[0] = o;
    c.data[1] = ot;
    if (!ot || ow == otw) return run(ow, ot ? 2 : 1);
    run(ow, 1);
    c.data[0] = ot;
    run(otw, 1);
}

}  // namespace ahead

namespace ahead {
// ANhelper<V>::mulIfEncoded(x, f) on the host with f = the column's A^-1:
// (storage)(x * A^-1) for an encoded column, (storage)x otherwise.  Used for
// re-encoding factors A_new * A_old^-1 (hashjoinAN.tcc:95-96, matchjoinAN.tcc:80-81).
inline uint64_t dec_if_host(const DCol& c, uint64_t x) { return c.enc ? mulw(x, c.ainv, c.width) : (x & wmask(c.width)); }
}  // namespace ahead
