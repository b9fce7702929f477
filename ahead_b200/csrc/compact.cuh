// compact.cuh -- stable multi-stream compaction in streaming passes.
//
// Every AN operator that filters rows (selectAN, checkAndDecodeAN, the
// positional matchjoinAN / fetchjoinAN ...) produces up to five output
// streams in scan order: the kept rows (stream 0, dense) and up to four
// error-position vectors (rare).  The reference builds them with push_back in
// one sequential loop (e.g. lib/column_operators/AN/selectAN_scalar.tcc:84-92).
//
// The unit of work is a tile of 32 * K rows that one warp owns in every pass,
// so no pass waits on another warp:
//   pass 1  classify: a lane reads 16-byte vectors of consecutive rows, sets a
//           bit per row of stream 0 in a register of its own, and three or so
//           shuffles turn the lanes' bits into row-ordered bitmap words.  A
//           vector's registers take the next load as soon as its rows have been
//           evaluated, so that loads are always in flight.
//   pass 2  scan: the per-tile counts become offsets (blocks of 1024 tiles; the
//           last block to finish scans the group totals).
//   pass 3  emit: the warp lists its kept rows in shared memory and writes
//           stream 0 with consecutive lanes on consecutive positions; a tile
//           whose every row is kept is a plain transform; the sparse streams are
//           recomputed only for tiles that hold any.
// Up to 32 small tiles one block does all three in one launch.
//
// K is 32 for long columns (fewest instructions per row) and 8 below 2^23 rows
// (enough warps to fill the chip) and for operators whose every row waits on a
// gather.  Measured on 600M 32-bit codes, a fifth selected: classify 367 us, the
// copy bandwidth (2.4 GB; 459 us with a ballot per 32 rows, 20 instructions a
// row instead of 8, and 450 fed through a shared-memory ring); emit 243 us for
// 0.96 GB (660 us when a block walked 4096-row tiles without looking ahead): it
// is bound by its ~380 instructions per 1024 rows.  Traffic beyond the input and the outputs: one bit per row, and 20
// bytes per tile and stream, written and read back, plus re-reading the few
// tiles with errors.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace ahead {

constexpr int kCThreads = 256;  // threads per block
constexpr int kCWarps = kCThreads / 32;
constexpr uint64_t kLongColumn = 1ull << 23;  // rows from which tiles are long
constexpr uint32_t kOneBlockTiles = 32;       // up to here one block runs the whole compaction

// Rows per lane of a tile: long ones, and short ones (at least one 16-byte vector).
constexpr int kLongK = 32;
constexpr int short_k(int w) { return w == 1 ? 16 : 8; }
template <class Op>
AHEAD_HD constexpr bool long_tiles(uint64_t n) {
    return !Op::GATHER && n >= kLongColumn;
}
template <class Op>
inline uint32_t compact_tiles(uint64_t n) {
    const uint64_t r = 32 * (long_tiles<Op>(n) ? kLongK : short_k(Op::W));
    return (uint32_t)((n + r - 1) / r);
}

template <int W>
AHEAD_DEV uint64_t gmem_ld(const char* p, uint64_t i) {
    if (W == 1) return __ldg((const uint8_t*)p + i);
    if (W == 2) return __ldg((const uint16_t*)p + i);
    if (W == 4) return __ldg((const uint32_t*)p + i);
    return __ldg((const unsigned long long*)p + i);
}

// Scratch of one compaction: bitmap words, per-tile counts and offsets.
struct CompactBufs {
    uint32_t* words;    // [ntiles * K] stream-0 bitmap
    uint32_t* counts;   // [ntiles][NCH]
    uint64_t* offsets;  // [ntiles][NCH] exclusive offset within the tile's group
    uint64_t* gbase;    // [ngroups][NCH] exclusive offset of each group of 1024 tiles
    uint64_t* totals;   // [NCH]
    uint32_t* done;     // blocks of the scan that have finished; zero between scans
    uint32_t ntiles;
    uint32_t nchan;
};

constexpr int kScanGroup = 1024;  // tiles per first-level scan block

AHEAD_HD uint32_t scan_groups(uint32_t ntiles) { return (ntiles + kScanGroup - 1) / kScanGroup; }

inline size_t compact_bytes(uint64_t n, uint32_t ntiles, uint32_t nchan) {
    return (size_t)(n + 1023) / 1024 * 128 + (size_t)ntiles * nchan * 12 + (size_t)scan_groups(ntiles) * nchan * 8 +
           4096;
}

// `Op` supplies
//   static constexpr int W;     width in bytes of the driving column `base`
//   static constexpr int NCH;   number of output streams (0 = kept rows)
//   static constexpr bool ACC;  sum the eval accumulator into *op.acc
//   static constexpr bool GATHER; eval loads from other places than row `row`
//   static constexpr bool EMIT_V; stream 0 emission needs the driving value
//   static constexpr int NOUT;  output columns written per stream-0 row
//   const char* base;
//   uint32_t eval(uint64_t v, uint64_t row, uint64_t& acc) const;  bit c = stream c
//   uint64_t out0(int k, uint64_t v, uint64_t row) const;  k-th output of a kept row
//   uint64_t cap0() const;      positions below it are stored
//   void* optr(int k) const; int owidth(int k) const;  where, and how wide, or instead
//   void put0(int k, uint64_t pos, uint64_t val) const;    store it at pos < cap0()
//   void rows0(v[U], row0, idx[U], val[NOUT][U]) const;    optional: the outputs of U kept
//                               rows row0 + idx[u] at once, so that their loads overlap
//   void emit(int c, uint64_t pos, uint64_t v, uint64_t row) const;  streams c >= 1, if there are any
//
//   void begin();  optional: loads what eval and out0 need from device memory, once per thread
//   void tile(uint32_t t);  optional: the same for each tile, before its rows
//
// Row layout of a tile: with VEC = 16 / W rows per vector, lane l holds in
// vector s the rows 32 * VEC * s + VEC * l + (0 .. VEC - 1) of the tile.

template <class Op>
AHEAD_DEV auto begin_op(Op& op, int) -> decltype(op.begin(), void()) {
    op.begin();
}
template <class Op>
AHEAD_DEV void begin_op(Op&, long) {}
template <class Op>
AHEAD_DEV auto begin_tile(Op& op, uint32_t tile, int) -> decltype(op.tile(tile), void()) {
    op.tile(tile);
}
template <class Op>
AHEAD_DEV void begin_tile(Op&, uint32_t, long) {}

template <int W>
AHEAD_DEV void unpack16(const uint4 q, uint64_t (&v)[16 / W]) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 16 / W; ++k) {
        if (W == 8) v[k] = (uint64_t)w[2 * k] | ((uint64_t)w[2 * k + 1] << 32);
        else if (W == 4) v[k] = w[k];
        else if (W == 2) v[k] = (w[k / 2] >> (16 * (k & 1))) & 0xffffu;
        else v[k] = (w[k / 4] >> (8 * (k & 3))) & 0xffu;
    }
}

// The vectors a lane has in flight: half a long tile, all of a short one.
template <int W, int K>
struct Flight {
    static constexpr int VEC = 16 / W;
    static constexpr int NV = K / VEC;                       // vectors per tile
    static constexpr int NF = NV > 1 && K == kLongK ? NV / 2 : NV;  // in flight
    uint4 q[NF];
    AHEAD_DEV static uint4 get(const char* base, uint64_t row, bool vec) {
        if (vec) return __ldg(reinterpret_cast<const uint4*>(base + row * W));
        uint32_t w[4] = {0, 0, 0, 0};  // a column that starts off a 16-byte boundary
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
            const uint64_t x = gmem_ld<W>(base, row + k);
            if (W == 8) {
                w[2 * k] = (uint32_t)x;
                w[2 * k + 1] = (uint32_t)(x >> 32);
            } else {
                w[k * W / 4] |= (uint32_t)x << (8 * (k * W % 4));
            }
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
    AHEAD_DEV void load(const char* base, uint64_t row, bool vec) {
#pragma unroll
        for (int s = 0; s < NF; ++s) q[s] = get(base, row + 32 * VEC * s, vec);
    }
};

// Lanes' bits to row-ordered words.  Bit VEC * s + q of lane l's `bits` is row
// 32 * VEC * s + VEC * l + q, so swapping the lane's low bits with s leaves the
// word of 32 rows number (32 / LPW) * s + l / LPW, LPW = 32 / VEC lanes a word, in
// lane LPW * (l / LPW) + s; a last shuffle brings word w to lane w.
template <int VEC>
AHEAD_DEV uint32_t words_of(uint32_t bits) {
    constexpr int LPW = 32 / VEC;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < LPW; d <<= 1) {
        const int j = VEC * d;  // the bit distance that lane distance d swaps with
        // positions whose index has bit j clear
        constexpr uint32_t all = 0xffffffffu;
        const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : all;
        const uint32_t o = __shfl_xor_sync(kFull, bits, d);
        bits = (lane & d) ? ((bits & ~m) | ((o >> j) & m)) : ((bits & m) | ((o & m) << j));
    }
    if (LPW == 1) return bits;
    // word w = VEC * s + h (h = lane / LPW) sits in lane LPW * h + s
    return __shfl_sync(kFull, bits, LPW * (lane % VEC) + lane / VEC);
}

// One tile's stream-0 words (lane s < K returns word s) and its counts (lane c
// returns stream c's).  A whole tile's first vectors are in `f`; the tile
// `next` (0: none) is loaded as registers free up.
template <class Op, int K>
AHEAD_DEV void tile_classify(const Op& op, uint64_t n, uint32_t tile, Flight<Op::W, K>& f, uint32_t next, bool vec,
                             uint64_t& acc, uint32_t& word, uint32_t& count) {
    typedef Flight<Op::W, K> F;
    constexpr int VEC = F::VEC;
    constexpr int NCH = Op::NCH;
    const int lane = threadIdx.x & 31;
    const uint64_t row0 = (uint64_t)tile * (32 * K) + VEC * lane;
    uint32_t mine = 0, sparse[NCH];
#pragma unroll
    for (int c = 0; c < NCH; ++c) sparse[c] = 0;
    auto take = [&](uint32_t bits, int at) {
        if (bits & 1u) mine |= 1u << at;
#pragma unroll
        for (int c = 1; c < NCH; ++c)
            if (bits & (1u << c)) ++sparse[c];
    };
    if ((uint64_t)(tile + 1) * (32 * K) <= n) {
#pragma unroll
        for (int s = 0; s < F::NV; ++s) {
            const uint64_t row = row0 + 32 * VEC * s;
            uint64_t v[VEC];
            unpack16<Op::W>(f.q[s % F::NF], v);
            if (s + F::NF < F::NV) f.q[s % F::NF] = F::get(op.base, row + 32 * VEC * F::NF, vec);
            else if (next)
                f.q[s % F::NF] = F::get(op.base, (uint64_t)next * (32 * K) + VEC * lane + 32 * VEC * (s % F::NF), vec);
#pragma unroll
            for (int q = 0; q < VEC; ++q) take(op.eval(v[q], row + q, acc), VEC * s + q);
        }
    } else {
#pragma unroll
        for (int s = 0; s < F::NV; ++s)
            for (int q = 0; q < VEC; ++q) {
                const uint64_t row = row0 + 32 * VEC * s + q;
                if (row < n) take(op.eval(gmem_ld<Op::W>(op.base, row), row, acc), VEC * s + q);
            }
    }
    word = words_of<VEC>(mine);
    count = __reduce_add_sync(kFull, (uint32_t)__popc(mine));
#pragma unroll
    for (int c = 1; c < NCH; ++c) {
        const uint32_t t = __reduce_add_sync(kFull, sparse[c]);
        if (lane == c) count = t;
    }
}

// U rows' values of one column, at row0 + idx[u] or (gather) at p[u]: the type is
// the same for all, so its branches are taken once for the U loads.
template <int U>
AHEAD_DEV void load_rows(const DCol& c, uint64_t row0, const uint32_t (&idx)[U], uint64_t (&x)[U]) {
    if (c.type == AHEAD_VOID) {
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = (uint32_t)(c.seqbase + row0 + idx[u]);
        return;
    }
    auto ld = [&](auto* p) {
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = __ldg(p + row0 + idx[u]);
    };
    if (c.width == 8) ld((const unsigned long long*)c.data);
    else if (c.width == 4) ld((const uint32_t*)c.data);
    else if (c.width == 2) ld((const uint16_t*)c.data);
    else ld((const uint8_t*)c.data);
}
template <int U>
AHEAD_DEV void gather_rows(const DCol& c, const uint64_t (&p)[U], uint64_t (&x)[U]) {
    if (c.type == AHEAD_VOID) {
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = (uint32_t)(c.seqbase + p[u]);
        return;
    }
    auto ld = [&](auto* d) {
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = __ldg(d + p[u]);
    };
    if (c.width == 8) ld((const unsigned long long*)c.data);
    else if (c.width == 4) ld((const uint32_t*)c.data);
    else if (c.width == 2) ld((const uint16_t*)c.data);
    else ld((const uint8_t*)c.data);
}

template <class Op, class V, int U>
AHEAD_DEV auto outputs_of(const Op& op, const V (&v)[U], uint64_t row0, const uint32_t (&idx)[U],
                          uint64_t (&val)[Op::NOUT][U], int) -> decltype(op.rows0(v, row0, idx, val), void()) {
    op.rows0(v, row0, idx, val);
}
template <class Op, class V, int U>
AHEAD_DEV void outputs_of(const Op& op, const V (&v)[U], uint64_t row0, const uint32_t (&idx)[U],
                          uint64_t (&val)[Op::NOUT][U], long) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int o = 0; o < Op::NOUT; ++o) val[o][u] = op.out0(o, v[u], row0 + idx[u]);
}

// Outputs u go to position base + i0 + 32 * u while i0 + 32 * u < room.
template <class Op, int U>
AHEAD_DEV auto store_outputs(const Op& op, uint64_t base, uint32_t i0, uint32_t room, const uint64_t (&val)[Op::NOUT][U],
                             int) -> decltype(op.optr(0), void()) {
#pragma unroll
    for (int o = 0; o < Op::NOUT; ++o) {
        auto st = [&](auto* p) {
            p += base + i0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i0 + 32 * u < room) p[32 * u] = val[o][u];
        };
        const int w = op.owidth(o);
        if (w == 8) st((uint64_t*)op.optr(o));
        else if (w == 4) st((uint32_t*)op.optr(o));
        else if (w == 2) st((uint16_t*)op.optr(o));
        else st((uint8_t*)op.optr(o));
    }
}
template <class Op, int U>
AHEAD_DEV void store_outputs(const Op& op, uint64_t base, uint32_t i0, uint32_t room, const uint64_t (&val)[Op::NOUT][U],
                             long) {
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (i0 + 32 * u < room) {
#pragma unroll
            for (int o = 0; o < Op::NOUT; ++o) op.put0(o, base + i0 + 32 * u, val[o][u]);
        }
}

// Writes one tile's stream-0 rows to positions base, base + 1, ...: lane s < K
// holds word s, `cnt` rows are kept, `list` is this warp's 32 * K half-words of
// shared memory.  Four rows per lane are in flight at a time, since an output
// may be a chain of gathers.
template <class Op, int K>
AHEAD_DEV void tile_emit(const Op& op, uint64_t n, uint32_t tile, uint32_t word, uint32_t cnt, uint64_t base,
                         uint16_t* list) {
    constexpr int W = Op::W;
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    const uint64_t trow0 = (uint64_t)tile * (32 * K);
    const uint32_t trows = trow0 + 32 * K <= n ? (uint32_t)(32 * K) : (uint32_t)(n - trow0);
    const bool all = cnt == trows;  // every row: position i is row i
    if (!all) {  // lane l lists the kept ones of rows [K * l, K * l + K), the last one first
        uint32_t h = word;
        if (K < 32) h = (__shfl_sync(kFull, word, lane * K / 32) >> (lane * K % 32)) & ((1u << (K & 31)) - 1u);
        uint16_t* at = list + warp_incl_scan(__popc(h));
        while (h) {
            const uint32_t b = 31 - __clz(h);
            *--at = (uint16_t)(K * lane + b);
            h ^= 1u << b;
        }
        __syncwarp();
    }
    const uint64_t fit = op.cap0() > base ? op.cap0() - base : 0;  // positions that are stored
    const uint32_t room = fit < cnt ? (uint32_t)fit : cnt;
    const uint32_t spare = all ? 0 : list[0];  // a kept row, for the lanes past the last one
    for (uint32_t i0 = lane; i0 < cnt; i0 += 32 * U) {
        uint32_t idx[U];
        uint64_t val[Op::NOUT][U];
        typename std::conditional<W == 8, uint64_t, uint32_t>::type v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = i0 + 32 * u;
            idx[u] = i < cnt ? (all ? i : list[i]) : spare;
            v[u] = Op::EMIT_V ? gmem_ld<W>(op.base + trow0 * W, idx[u]) : 0;
        }
        outputs_of(op, v, trow0, idx, val, 0);
        store_outputs(op, base, i0, room, val, 0);
    }
    if (!all) __syncwarp();  // the list is reused
}

// Writes one tile's sparse streams: lane c holds stream c's count and position.
// Four loads in flight: one warp walks the whole tile, and a load at a time made
// these tiles the emit pass's tail (30M 8-byte codes, 1,000 of them corrupt: emit 30
// us, 57 before, 17 without errors).
template <class Op, int K>
AHEAD_DEV void tile_emit_sparse(const Op& op, uint64_t n, uint32_t tile, uint64_t base) {
    constexpr int W = Op::W;
    const int lane = threadIdx.x & 31;
    const uint64_t row0 = (uint64_t)tile * (32 * K) + lane;
    uint64_t pos[Op::NCH];
#pragma unroll
    for (int c = 1; c < Op::NCH; ++c) pos[c] = __shfl_sync(kFull, base, c);
    uint64_t dummy = 0;
    constexpr int U = 4;  // loads in flight
    uint64_t v[U];
#pragma unroll 1
    for (int s0 = 0; s0 < K; s0 += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t row = row0 + 32 * (s0 + u);
            v[u] = row < n ? gmem_ld<W>(op.base, row) : 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t row = row0 + 32 * (s0 + u);
            const uint32_t bits = row < n ? op.eval(v[u], row, dummy) : 0u;
            if (!__any_sync(kFull, bits > 1u)) continue;
#pragma unroll
            for (int c = 1; c < Op::NCH; ++c) {
                const uint32_t b = __ballot_sync(kFull, (bits >> c) & 1u);
                if ((bits >> c) & 1u) op.emit(c, pos[c] + __popc(b & ((1u << lane) - 1u)), v[u], row);
                pos[c] += __popc(b);
            }
        }
    }
}

// Pass 1, `per` tiles per warp.
template <class Op, int K>
__global__ void __launch_bounds__(kCThreads) classify_kernel(Op op, uint64_t n, CompactBufs cb, int per) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec = ((uintptr_t)op.base & 15) == 0;
    begin_op(op, 0);
    uint64_t acc = 0;
    const uint32_t whole = (uint32_t)(n / (32 * K));  // whole tiles
    uint32_t tile = blockIdx.x * per * kCWarps + warp;
    Flight<Op::W, K> f;
    if (tile < whole) f.load(op.base, (uint64_t)tile * (32 * K) + 16 / Op::W * lane, vec);
    for (int k = 0; k < per && tile < cb.ntiles; ++k, tile += kCWarps) {
        const uint32_t next = k + 1 < per && tile + kCWarps < whole ? tile + kCWarps : 0;
        uint32_t word, count;
        begin_tile(op, tile, 0);
        tile_classify<Op, K>(op, n, tile, f, next, vec, acc, word, count);
        if (lane < K) cb.words[(size_t)tile * K + lane] = word;
        if (lane < Op::NCH) cb.counts[(size_t)tile * Op::NCH + lane] = count;
    }
    if constexpr (Op::ACC) {
        acc = warp_sum64(acc);
        if (lane == 0 && acc) atomicAdd((unsigned long long*)op.acc, (unsigned long long)acc);
    }
}

// Exclusive scan of one value per thread over a block of 1024; *total by every thread.
AHEAD_DEV uint64_t block_scan_1024(uint64_t x, uint64_t* s_part, uint64_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t incl = warp_incl_scan64(x);
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint64_t p = s_part[lane];
        const uint64_t pi = warp_incl_scan64(p);
        s_part[lane] = pi - p;
        if (lane == 31) s_part[32] = pi;
    }
    __syncthreads();
    const uint64_t r = s_part[warp] + incl - x;
    *total = s_part[32];
    __syncthreads();
    return r;
}

// The group totals in gbase to exclusive group offsets, by one block of 1024: a
// warp per stream while they are few.
AHEAD_DEV void scan_group_totals(const CompactBufs& cb, uint64_t* s_part) {
    const uint32_t nch = cb.nchan, ng = scan_groups(cb.ntiles), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (ng <= 128) {
        if (warp >= nch) return;
        uint64_t carry = 0;
        for (uint32_t g0 = 0; g0 < ng; g0 += 32) {
            const uint32_t g = g0 + lane;
            uint64_t* p = cb.gbase + (size_t)g * nch + warp;
            const uint64_t x = g < ng ? __ldcg((const unsigned long long*)p) : 0;
            const uint64_t incl = warp_incl_scan64(x);
            if (g < ng) *p = carry + incl - x;
            carry += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0) cb.totals[warp] = carry;
        return;
    }
    for (uint32_t c = 0; c < nch; ++c) {
        uint64_t carry = 0;
        for (uint32_t g0 = 0; g0 < ng; g0 += kScanGroup) {
            const uint32_t g = g0 + threadIdx.x;
            const uint64_t x = g < ng ? __ldcg((const unsigned long long*)&cb.gbase[(size_t)g * nch + c]) : 0;
            uint64_t total;
            const uint64_t ex = block_scan_1024(x, s_part, &total);
            if (g < ng) cb.gbase[(size_t)g * nch + c] = carry + ex;
            carry += total;
        }
        if (threadIdx.x == 0) cb.totals[c] = carry;
    }
}

// Pass 2: each block scans the counts of 1024 consecutive tiles per stream
// (exclusive, within the group; three streams' counts of at most 1024 share a
// 64-bit word, 21 bits each) and writes the group totals to gbase; the last
// block to finish turns those into exclusive group offsets.  (As two kernels, each
// scanning stream after stream, this took 10-14 us of every operator with up to a
// few thousand tiles.)  From kScanSplit groups on -- the slots of a large hash table,
// compactions of 2^28 rows in short tiles or 2^30 in long ones -- the offsets get a
// launch of their own: each block's fence and count took 96 us of 8M slots, 55 without.
constexpr uint32_t kScanSplit = 1024;

static __global__ void __launch_bounds__(kScanGroup) group_scan_kernel(CompactBufs cb) {
    __shared__ uint64_t s_part[33];
    scan_group_totals(cb, s_part);
}

static __global__ void __launch_bounds__(kScanGroup) tile_scan_kernel(CompactBufs cb) {
    __shared__ uint64_t s_part[33];
    __shared__ bool s_last;
    const uint32_t nch = cb.nchan, ng = scan_groups(cb.ntiles);
    const uint32_t t = blockIdx.x * kScanGroup + threadIdx.x;
    for (uint32_t c0 = 0; c0 < nch; c0 += 3) {
        const uint32_t m = nch - c0 < 3 ? nch - c0 : 3;
        const uint64_t part = m == 1 ? ~0ull : (1ull << 21) - 1;  // (a single stream's counts may be larger)
        uint64_t x = 0;
        if (t < cb.ntiles)
            for (uint32_t c = 0; c < m; ++c) x |= (uint64_t)cb.counts[(size_t)t * nch + c0 + c] << (21 * c);
        uint64_t total;
        const uint64_t ex = block_scan_1024(x, s_part, &total);
        if (t < cb.ntiles)
            for (uint32_t c = 0; c < m; ++c) cb.offsets[(size_t)t * nch + c0 + c] = (ex >> (21 * c)) & part;
        if (threadIdx.x < m) {
            const uint64_t tot = (total >> (21 * threadIdx.x)) & part;
            cb.gbase[(size_t)blockIdx.x * nch + c0 + threadIdx.x] = ng == 1 ? 0 : tot;
            if (ng == 1) cb.totals[c0 + threadIdx.x] = tot;
        }
    }
    if (ng == 1 || ng >= kScanSplit) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(cb.done, 1u) == gridDim.x - 1;
        if (s_last) *cb.done = 0;
        __threadfence();
    }
    __syncthreads();
    if (s_last) scan_group_totals(cb, s_part);
}

// Launches pass 2; returns the number of launches.
inline int scan_tiles(cudaStream_t st, const CompactBufs& cb) {
    const uint32_t ng = scan_groups(cb.ntiles);
    tile_scan_kernel<<<ng, kScanGroup, 0, st>>>(cb);
    if (ng < kScanSplit) return 1;
    group_scan_kernel<<<1, kScanGroup, 0, st>>>(cb);
    return 2;
}

// Pass 3, `per` tiles per warp; the next tile's header and words are loaded
// before this one's rows are written.
template <class Op, int K>
__global__ void __launch_bounds__(kCThreads) emit_kernel(Op op, uint64_t n, CompactBufs cb, int per) {
    constexpr int NCH = Op::NCH;
    __shared__ uint16_t s_rows[kCWarps][32 * K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    begin_op(op, 0);
    auto tile_of = [&](int k) { return (blockIdx.x * per + k) * kCWarps + warp; };
    uint32_t word = 0, count = 0;
    uint64_t base = 0;
    auto head = [&](uint32_t tile) {
        word = count = 0;
        base = 0;
        if (tile >= cb.ntiles) return;
        if (lane < K) word = __ldg(cb.words + (size_t)tile * K + lane);
        if (lane < NCH) {
            count = __ldg(cb.counts + (size_t)tile * NCH + lane);
            base = __ldg((const unsigned long long*)cb.offsets + (size_t)tile * NCH + lane) +
                   __ldg((const unsigned long long*)cb.gbase + (size_t)(tile / kScanGroup) * NCH + lane);
        }
    };
    head(tile_of(0));
    for (int k = 0; k < per; ++k) {
        const uint32_t tile = tile_of(k);
        if (tile >= cb.ntiles) break;
        const uint32_t w = word, c = count;
        const uint64_t b = base;
        if (k + 1 < per) head(tile_of(k + 1));
        const uint32_t c0 = __shfl_sync(kFull, c, 0);
        begin_tile(op, tile, 0);
        if (c0) tile_emit<Op, K>(op, n, tile, w, c0, __shfl_sync(kFull, b, 0), s_rows[warp]);
        if constexpr (NCH > 1)
            if (__any_sync(kFull, lane > 0 && c)) tile_emit_sparse<Op, K>(op, n, tile, b);
    }
}

// All passes in one block, for up to kOneBlockTiles short tiles: warp w owns tile w.
template <class Op>
__global__ void __launch_bounds__(kOneBlockTiles * 32) compact_one_kernel(Op op, uint64_t n, CompactBufs cb) {
    constexpr int NCH = Op::NCH;
    constexpr int K = short_k(Op::W);
    __shared__ uint16_t s_rows[kOneBlockTiles][32 * K];
    __shared__ uint32_t s_cnt[NCH][kOneBlockTiles];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec = ((uintptr_t)op.base & 15) == 0;
    begin_op(op, 0);
    uint32_t word = 0, count = 0;
    uint64_t acc = 0;
    Flight<Op::W, K> f;
    if ((uint64_t)(warp + 1) * (32 * K) <= n) f.load(op.base, (uint64_t)warp * (32 * K) + 16 / Op::W * lane, vec);
    begin_tile(op, warp, 0);
    tile_classify<Op, K>(op, n, warp, f, 0, vec, acc, word, count);
    if (lane < NCH) s_cnt[lane][warp] = count;
    __syncthreads();
    uint64_t base = 0;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const uint32_t x = lane < (int)(blockDim.x >> 5) ? s_cnt[c][lane] : 0;
        const uint32_t before = __reduce_add_sync(kFull, lane < warp ? x : 0u);
        const uint32_t total = __reduce_add_sync(kFull, x);
        if (lane == c) base = before;
        if (threadIdx.x == 0) cb.totals[c] = total;
    }
    const uint32_t c0 = __shfl_sync(kFull, count, 0);
    if (c0) tile_emit<Op, K>(op, n, warp, word, c0, __shfl_sync(kFull, base, 0), s_rows[warp]);
    if constexpr (NCH > 1)
        if (__any_sync(kFull, lane > 0 && lane < NCH && count)) tile_emit_sparse<Op, K>(op, n, warp, base);
    if constexpr (Op::ACC) {
        acc = warp_sum64(acc);
        if (lane == 0 && acc) atomicAdd((unsigned long long*)op.acc, (unsigned long long)acc);
    }
}

}  // namespace ahead
