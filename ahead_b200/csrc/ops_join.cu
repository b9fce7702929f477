// ops_join.cu -- hashjoinAN / hashjoin, matchjoinAN / matchjoin and
// fetchjoinAN / fetchjoin.
//
// Hash joins key the build side (the right BAT by default) by its decoded keys
// cast to the unencoded base type, probe in probe-row order and emit every match
// in build order (lib/column_operators/AN/hashjoinAN.tcc:54-223).  Unique keys
// of a bounded range (a dimension's keys) index a bitmap and a value array
// directly, and the probe is a compaction; anything else, and a call with too
// little device memory for these, takes the hash table of hash.cuh.  Rows with
// detected errors are still built and probed, exactly as in the reference; the
// four error vectors are checks of the four inputs.
//
// Positional match/fetch joins (matchjoinAN.tcc:226-354) gather once per OID,
// write every row to its own place and close the gaps of the few rows they drop;
// short lists, many dropped rows and short device memory take a compaction over
// the list.  The merge matchjoin (matchjoinAN.tcc:46-144) is an intersection when
// the keys of both inputs strictly increase (the common case: two selection
// vectors), with the error positions of corrupt values derived per row; keys out
// of order replay the reference's merge loop step by step on the device, so that
// every error push (including its repeated checks of the same row) is reproduced.
#include "hash.cuh"
#include "ops_common.cuh"

using namespace ahead;

namespace {

// --------------------------------------------------------------- hash join
struct KeyCfg {
    DCol col;
    uint64_t ainv, keymask, largermask, condmax;
    int dec, width;
};

AHEAD_DEV bool key_of(const KeyCfg& k, uint64_t row, uint64_t& key) {
    const uint64_t v = load_at(k.col, row);
    const uint64_t d = k.dec ? mulw(v, k.ainv, k.width) : v;
    if ((d & k.largermask) > k.condmax) return false;
    key = d & k.keymask;
    return true;
}

__global__ void ht_build_kernel(HashTab h, KeyCfg kc, uint64_t n, uint32_t* slot_of) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t key = 0;
        key_of(kc, i, key);
        const uint32_t s = ht_insert(h, key);
        slot_of[i] = s;
        atomicAdd(&h.cnt[s], 1u);
    }
}

__global__ void ht_offsets_kernel(HashTab h, CompactBufs cb) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < cb.ntiles; s += gridDim.x * blockDim.x)
        h.off[s] = (uint32_t)(cb.offsets[s] + cb.gbase[s / kScanGroup]);
}

__global__ void ht_fill_kernel(HashTab h, const uint32_t* slot_of, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = slot_of[i];
        h.rows[h.off[s] + atomicAdd(&h.cur[s], 1u)] = (uint32_t)i;
    }
}

// Restore build order inside the (rare) segments with several rows.
__global__ void ht_order_kernel(HashTab h, uint32_t nslots) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x) {
        const uint32_t c = h.cnt[s];
        if (c < 2) continue;
        uint32_t* r = h.rows + h.off[s];
        for (uint32_t i = 1; i < c; ++i) {
            const uint32_t x = r[i];
            uint32_t j = i;
            while (j > 0 && r[j - 1] > x) {
                r[j] = r[j - 1];
                --j;
            }
            r[j] = x;
        }
    }
}

struct JoinOut {
    DCol pcol, bcol;  // probe-side and build-side output columns
    uint64_t fh, ft, cap;
    void *oh, *ot;
    int probe_is_head, rh, rt, ohw, otw;
};

AHEAD_DEV void join_emit(const JoinOut& o, uint64_t pos, uint64_t prow, uint64_t brow) {
    if (pos >= o.cap) return;
    uint64_t hv = o.probe_is_head ? load_at(o.pcol, prow) : load_at(o.bcol, brow);
    uint64_t tv = o.probe_is_head ? load_at(o.bcol, brow) : load_at(o.pcol, prow);
    if (o.rh) hv *= o.fh;
    if (o.rt) tv *= o.ft;
    store_at(o.oh, o.ohw, pos, hv);
    store_at(o.ot, o.otw, pos, tv);
}

constexpr int kProbeRowsPerThread = 16;
constexpr int kProbeTile = 256 * kProbeRowsPerThread;  // probe rows per block and step
// a probe row's entry: kNoSlot, the single matching build row | kDirect, or
// the slot of a key with several build rows
constexpr uint32_t kDirect = 0x80000000u;

// the packed probe table (after the build's order step)
__global__ void ht_pack_kernel(HashTab h, ProbeSlot* t, uint32_t nslots, bool direct) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x) {
        ProbeSlot e;
        e.key = h.keys[s];
        e.cnt = h.cnt[s];
        e.first = (direct && e.cnt == 1) ? h.rows[h.off[s]] : h.off[s];
        t[s] = e;
    }
}

// Pass A: find every probe row's slot and count its matches per tile.
__global__ void __launch_bounds__(256) probe_count_kernel(const ProbeSlot* __restrict__ pt, uint32_t mask, bool direct,
                                                          KeyCfg pk, uint64_t n, uint32_t* pslot, CompactBufs cb) {
    __shared__ uint32_t s_w[8];
    for (uint32_t tile = blockIdx.x; tile < cb.ntiles; tile += gridDim.x) {
        uint32_t c = 0;
#pragma unroll 4
        for (int k = 0; k < kProbeRowsPerThread; ++k) {
            const uint64_t row = (uint64_t)tile * kProbeTile + k * 256 + threadIdx.x;
            if (row >= n) break;
            uint64_t key = 0;
            uint32_t s = kNoSlot;
            ProbeSlot e;
            if (key_of(pk, row, key)) s = ps_find(pt, mask, key, e);
            if (s != kNoSlot) {
                c += e.cnt;
                if (direct && e.cnt == 1) s = e.first | kDirect;
            }
            pslot[row] = s;
        }
        c = __reduce_add_sync(kFull, c);
        if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (int w = 0; w < 8; ++w) t += s_w[w];
            cb.counts[tile] = t;
        }
        __syncthreads();
    }
}

// Pass C: each thread owns 16 consecutive probe rows; a block scan of their
// match counts gives every row its output position.
__global__ void __launch_bounds__(256) probe_emit_kernel(const ProbeSlot* __restrict__ pt, const uint32_t* rows,
                                                         uint64_t n, const uint32_t* pslot, CompactBufs cb, JoinOut o) {
    __shared__ uint32_t s_w[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t tile = blockIdx.x; tile < cb.ntiles; tile += gridDim.x) {
        const uint64_t r0 = (uint64_t)tile * kProbeTile + (uint64_t)threadIdx.x * kProbeRowsPerThread;
        uint32_t c = 0;
        for (int k = 0; k < kProbeRowsPerThread; ++k) {
            const uint64_t row = r0 + k;
            if (row >= n) break;
            const uint32_t s = pslot[row];
            if (s != kNoSlot) c += (s & kDirect) ? 1u : pt[s].cnt;
        }
        const uint32_t incl = warp_incl_scan(c);
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        uint64_t pos = cb.offsets[tile] + cb.gbase[tile / kScanGroup] + incl - c;
        for (int w = 0; w < warp; ++w) pos += s_w[w];
        __syncthreads();
        if (!c) continue;
        for (int k = 0; k < kProbeRowsPerThread; ++k) {
            const uint64_t row = r0 + k;
            if (row >= n) break;
            const uint32_t s = pslot[row];
            if (s == kNoSlot) continue;
            if (s & kDirect) {
                join_emit(o, pos++, row, s & ~kDirect);
                continue;
            }
            const ProbeSlot e = pt[s];
            for (uint32_t j = 0; j < e.cnt; ++j) join_emit(o, pos++, row, rows[e.first + j]);
        }
    }
}

// --------------------------------------------------------- direct join
// A dimension's keys are unique and dense enough that key - smallest key can
// index an array: one bit says whether the key is there, one 8-byte word holds
// what the join emits for it (the build side's OID, re-encoded).  The probe is
// then a compaction of the probe rows whose bit is set -- a key has at most one
// match -- with the AN checks of the probe's columns as its sparse streams, so
// the probe column is read once per pass and nothing per row is stored between
// the passes.  The bitmap is copied into shared memory (up to kDjSmem bytes:
// 1.6M keys), where 32 lanes' lookups cost a few bank conflicts, not 32 L2
// requests; only the matches touch the value array in L2.
//
// Two things send the join to the hash table instead, found by the build
// kernels and read back with the counts: a key range above the limit (2^24 at
// most: the value array then stays near L2's size), or a repeated key.  The probe
// passes see it on the device and read nothing, which leaves some 40 us of
// launches ahead of the table (60M probe rows, one key of 320K repeated: 1.38 ms a
// call, 1.39 by the table alone; 30M against 3M keys of a wide range 1.95 and
// 1.92).  Not tried: more build rows than the limit, and 8-byte raw codes as
// keys (multiples of A: far too wide).
// At 60M probe rows against 320K of 800K keys: hash probe 512 + 559 us (one
// 16-byte slot request to L2 per row, then thread-serial output) and 110 us of
// separate column checks, against 15 us to build, 123 to classify and 219 to emit
// (DRAM floor of the two passes: 205).
constexpr uint64_t kDjMaxSpan = 1ull << 24;
constexpr int kDjSmem = 200 * 1024;
constexpr int kDjBounds = 20, kDjBad = 22, kDjBuildKey = 23, kDjBuildVal = 24, kDjCounters = 25;  // counters

inline uint64_t dj_limit(uint64_t nb, uint64_t np) {
    const uint64_t l = (1ull << 20) + 64 * nb + np;
    return (l < kDjMaxSpan ? l : kDjMaxSpan) & ~31ull;
}

// More rows than the range has keys: some key repeats.
inline bool dj_possible(uint64_t nb, uint64_t np) { return nb <= dj_limit(nb, np); }

struct DjBuild {
    KeyCfg bk;
    DCol bcol;        // build-side output column
    uint64_t nb, limit, factor;
    int reenc, check; // check: report corrupt keys and values
    uint64_t* bounds; // [0] the largest ~key, [1] the largest key
    uint32_t* bad;
    uint32_t* bits;   // [limit / 32]
    uint64_t* val;    // [limit]
    ErrList kerr, verr;
    AHEAD_DEV uint64_t kmin() const { return ~bounds[0]; }
    AHEAD_DEV uint64_t span() const { return bounds[1] - kmin() + 1; }
};

// Key bounds, the AN checks of the build columns, and the bitmap cleared.
__global__ void __launch_bounds__(256) dj_bounds_kernel(DjBuild b) {
    __shared__ uint64_t s_lo[8], s_hi[8];
    const uint64_t first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = first; w < b.limit / 32; w += stride) b.bits[w] = 0;
    uint64_t nlo = 0, hi = 0;
    for (uint64_t i = first; i < b.nb; i += stride) {
        const uint64_t v = load_at(b.bk.col, i);
        const uint64_t d = b.bk.dec ? mulw(v, b.bk.ainv, b.bk.width) : v;
        if (b.check && b.bk.col.enc && mulw(v, b.bk.col.ainv, b.bk.width) > b.bk.col.umax) b.kerr.add(i);
        if (b.check && b.bcol.enc && mulw(load_at(b.bcol, i), b.bcol.ainv, b.bcol.width) > b.bcol.umax) b.verr.add(i);
        const uint64_t k = d & b.bk.keymask;
        nlo = ~k > nlo ? ~k : nlo;
        hi = k > hi ? k : hi;
    }
    for (int d = 16; d > 0; d >>= 1) {
        const uint64_t a = __shfl_xor_sync(kFull, nlo, d), c = __shfl_xor_sync(kFull, hi, d);
        nlo = a > nlo ? a : nlo;
        hi = c > hi ? c : hi;
    }
    if ((threadIdx.x & 31) == 0) {
        s_lo[threadIdx.x >> 5] = nlo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            nlo = s_lo[w] > nlo ? s_lo[w] : nlo;
            hi = s_hi[w] > hi ? s_hi[w] : hi;
        }
        if (nlo) {  // (a block without rows holds 0)
            atomicMax((unsigned long long*)&b.bounds[0], (unsigned long long)nlo);
            atomicMax((unsigned long long*)&b.bounds[1], (unsigned long long)hi);
        }
    }
}

// Sets each key's bit and value.  Neighbouring lanes hold neighbouring keys
// (dimension tables are in key order), so the lanes of one word share one atomic.
// Once a key has repeated the warps stop, and no more of them write the word: 3M rows
// of 200K keys took 575 us with volatile reads of it next to every warp's write.
__global__ void __launch_bounds__(256) dj_insert_kernel(DjBuild b) {
    const uint64_t kmin = b.kmin(), span = b.span(), stride = (uint64_t)gridDim.x * blockDim.x;
    if (span > b.limit) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *b.bad = 1;
        return;
    }
    const uint64_t rounds = (b.nb + stride - 1) / stride;
    for (uint64_t r = 0; r < rounds; ++r) {
        if (__any_sync(kFull, ld_ca(b.bad) != 0)) return;  // (the hash table has the join)
        const uint64_t i = r * stride + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
        const bool live = i < b.nb;
        uint64_t d = 0;
        if (live) {
            const uint64_t v = load_at(b.bk.col, i);
            d = ((b.bk.dec ? mulw(v, b.bk.ainv, b.bk.width) : v) & b.bk.keymask) - kmin;
            const uint64_t x = load_at(b.bcol, i);
            b.val[d] = b.reenc ? x * b.factor : x;
        }
        const uint32_t word = live ? (uint32_t)(d >> 5) : ~0u, bit = live ? 1u << (d & 31) : 0u;
        const uint32_t peers = __match_any_sync(kFull, word);
        const uint32_t set = __reduce_or_sync(peers, bit);
        if (live && (threadIdx.x & 31) == __ffs(peers) - 1) {
            const uint32_t old = atomicOr(&b.bits[word], set);
            if (((old & set) || __popc(set) != __popc(peers)) && !ld_ca(b.bad)) *b.bad = 1;  // a key twice
        }
    }
}

// The probe.  Streams: 0 matching rows, 1 corrupt probe keys, 2 corrupt values
// of the probe side's output column.
template <int WW, bool AN>
struct DjOp {
    static constexpr int W = WW;
    static constexpr int NCH = AN ? 3 : 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = true;
    static constexpr bool EMIT_V = true;
    static constexpr int NOUT = 2;
    const char* base;
    KeyCfg pk;
    JoinOut o;
    const uint64_t* bounds;  // null: kmin and span are set
    const uint32_t* bad;
    const uint32_t* bits;
    const uint64_t* val;
    uint64_t limit;
    uint32_t kmin, span;  // set by begin (keys have at most 32 bits)
    uint64_t aoid, eck, eco;
    uint64_t *ek, *eo, *acc;
    AHEAD_DEV void begin() {
        if (!bounds) return;  // (known to the host by now)
        const uint64_t lo = ~__ldg((const unsigned long long*)bounds);
        const uint64_t m = __ldg((const unsigned long long*)bounds + 1) - lo + 1;
        kmin = (uint32_t)lo;
        span = (__ldg(bad) || m > limit) ? 0u : (uint32_t)m;
    }
    AHEAD_DEV uint64_t dec(uint64_t v) const { return pk.dec ? mulw(v, pk.ainv, W) : v; }
    AHEAD_DEV uint32_t key(uint64_t d) const { return ((uint32_t)d & (uint32_t)pk.keymask) - kmin; }
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t row, uint64_t&) const {
        const uint64_t d = dec(v);
        uint32_t b = 0;
        if (AN) {
            if (d > pk.col.umax) b |= 2u;
            if (o.pcol.enc && mulw(load_at(o.pcol, row), o.pcol.ainv, o.pcol.width) > o.pcol.umax) b |= 4u;
        }
        const uint32_t k = key(d);
        // (the key's range check only where the other side's keys are wider)
        if (pk.largermask > pk.condmax && (d & pk.largermask) > pk.condmax) return b;
        if (k < span && ((bits[k >> 5] >> (k & 31)) & 1u)) b |= 1u;
        return b;
    }
    // output 0: the probe side's value, output 1: the build side's
    template <class V, int U>
    AHEAD_DEV void rows0(const V (&v)[U], uint64_t row0, const uint32_t (&idx)[U], uint64_t (&x)[2][U]) const {
#pragma unroll
        for (int u = 0; u < U; ++u)
            x[1][u] = __ldg((const unsigned long long*)val + key(dec(v[u])));
        load_rows(o.pcol, row0, idx, x[0]);
        if (o.probe_is_head ? o.rh : o.rt) {
            const uint64_t f = o.probe_is_head ? o.fh : o.ft;
#pragma unroll
            for (int u = 0; u < U; ++u) x[0][u] *= f;
        }
    }
    AHEAD_DEV uint64_t cap0() const { return o.cap; }
    AHEAD_DEV void* optr(int k) const { return (k == 0) == (o.probe_is_head != 0) ? o.oh : o.ot; }
    AHEAD_DEV int owidth(int k) const { return (k == 0) == (o.probe_is_head != 0) ? o.ohw : o.otw; }
    AHEAD_DEV void emit(int c, uint64_t pos, uint64_t, uint64_t row) const {
        if (c == 1) {
            if (pos < eck) ek[pos] = row * aoid;
        } else if (pos < eco) {
            eo[pos] = row * aoid;
        }
    }
};

// Pass 1 with the bitmap in shared memory: one block of 32 warps per SM walks
// the tiles (a bitmap that does not fit is read through L1 and L2).
template <class Op>
__global__ void __launch_bounds__(1024, 1) dj_classify_kernel(Op op, uint64_t n, CompactBufs cb) {
    extern __shared__ uint32_t s_bits[];
    constexpr int K = short_k(Op::W);
    const int lane = threadIdx.x & 31;
    const bool vec = ((uintptr_t)op.base & 15) == 0;
    op.begin();
    const uint32_t whole = (uint32_t)(n / (32 * K)), nw = gridDim.x * 32;
    if (!op.span) {  // the hash table has the join: the probe column is not read, and no tile keeps a row
        const uint64_t words = (uint64_t)cb.ntiles * Op::NCH;
        for (uint64_t i = blockIdx.x * 1024ull + threadIdx.x; i < words; i += gridDim.x * 1024ull) cb.counts[i] = 0;
        return;
    }
    uint32_t tile = blockIdx.x * 32 + (threadIdx.x >> 5);
    Flight<Op::W, K> f;
    if (tile < whole) f.load(op.base, (uint64_t)tile * (32 * K) + 16 / Op::W * lane, vec);
    const uint32_t words = (uint32_t)((op.span + 31) / 32);
    if (words <= kDjSmem / 4) {
        for (uint32_t i = threadIdx.x; i < words; i += 1024) s_bits[i] = op.bits[i];
        __syncthreads();
        op.bits = s_bits;
    }
    uint64_t acc = 0;
    for (; tile < cb.ntiles; tile += nw) {
        const uint32_t next = tile + nw < whole ? tile + nw : 0;
        uint32_t word, count;
        tile_classify<Op, K>(op, n, tile, f, next, vec, acc, word, count);
        if (lane < K) cb.words[(size_t)tile * K + lane] = word;
        if (lane < Op::NCH) cb.counts[(size_t)tile * Op::NCH + lane] = count;
    }
}

size_t dj_scratch(uint64_t nb, uint64_t np) {
    const uint64_t limit = dj_limit(nb, np);
    return limit / 8 + limit * 8 + 2 * kErrListBytes + compact_scratch<DjOp<8, true>>(np) + 4096;
}

// Builds, probes and reads the counters back: counter 0 matches, 1 and 2 the
// probe's errors, kDjBad whether the hash table has to take the join.  `err_k`,
// `err_o`: the probe key's and the probe output column's vectors.  A sized call
// (`out` given) gets its output columns between the passes.
template <bool AN>
int run_direct_join(OpScope& s, const KeyCfg& bk, uint64_t nb, const KeyCfg& pk, uint64_t np, const JoinOut& o,
                    uint64_t aoid, ahead_errvec* err_k, ahead_errvec* err_o, ErrList* kerr, ErrList* verr,
                    ahead_bat* out) {
    cudaStream_t st = s.ctx->stream;
    DjBuild b;
    b.bk = bk;
    b.bcol = o.bcol;
    b.nb = nb;
    b.limit = dj_limit(nb, np);
    b.reenc = o.probe_is_head ? o.rt : o.rh;
    b.factor = o.probe_is_head ? o.ft : o.fh;
    b.check = AN;
    b.bounds = s.d_counters + kDjBounds;
    b.bad = (uint32_t*)(s.d_counters + kDjBad);
    b.bits = (uint32_t*)s.alloc(b.limit / 8);
    b.val = (uint64_t*)s.alloc(b.limit * 8);
    *kerr = b.kerr = err_list(s, kDjBuildKey);
    *verr = b.verr = err_list(s, kDjBuildVal);
    const uint64_t most = b.limit / 32 > nb ? b.limit / 32 : nb;
    const uint32_t g = (uint32_t)s.ctx->num_sms * 4, want = grid_for(most, 256);
    dj_bounds_kernel<<<want < g ? want : g, 256, 0, st>>>(b);
    dj_insert_kernel<<<grid_for(nb, 256), 256, 0, st>>>(b);
    s.launched(2);
    auto probe = [&](auto tag) -> int {
        typedef DjOp<decltype(tag)::value, AN> Op;
        Op op;
        op.base = (const char*)pk.col.data;
        op.pk = pk;
        op.o = o;
        op.bounds = b.bounds;
        op.bad = b.bad;
        op.bits = b.bits;
        op.val = b.val;
        op.limit = b.limit;
        op.kmin = op.span = 0;
        op.aoid = aoid;
        op.ek = edata(err_k);
        op.eo = edata(err_o);
        op.eck = ecap(err_k);
        op.eco = ecap(err_o);
        op.acc = nullptr;
        const uint32_t nt = compact_tiles<Op>(np);
        const CompactBufs cb = s.compact_bufs(np, nt, Op::NCH, 0);
        if (!out && nt <= kOneBlockTiles) {
            s.launched(launch_compact(s.ctx, st, op, np, cb));
            return s.finish(kDjCounters);
        }
        if (dyn_smem_ready<dj_classify_kernel<Op>>(s.ctx, kDjSmem)) {
            const uint32_t blocks = (nt + 31) / 32;
            dj_classify_kernel<Op><<<blocks < (uint32_t)s.ctx->num_sms ? blocks : s.ctx->num_sms, 1024, kDjSmem,
                                     st>>>(op, np, cb);
        } else {
            const uint32_t per = tiles_per_warp(s.ctx, nt);
            classify_kernel<Op, short_k(Op::W)>
                <<<(nt + per * kCWarps - 1) / (per * kCWarps), kCThreads, 0, st>>>(op, np, cb, (int)per);
        }
        s.launched();
        launch_scan(s, cb);
        if (out) {
            int rc = s.finish(kDjCounters);
            if (rc || s.counter(kDjBad)) return rc;
            // (finish() leaves the counters zero: the emit pass gets the key bounds by value)
            op.bounds = nullptr;
            op.kmin = (uint32_t)~s.counter(kDjBounds);
            op.span = (uint32_t)(s.counter(kDjBounds + 1) - ~s.counter(kDjBounds) + 1);
            op.o.cap = s.counter(0);
            if (!s.take(&out->head, 0, op.o.cap) || !s.take(&out->tail, 1, op.o.cap))
                return fail(s.ctx, AHEAD_NO_MEMORY, "output allocation failed");
            op.o.oh = out->head.data;
            op.o.ot = out->tail.data;
        }
        launch_emit(s, op, np, cb);
        return out ? s.wait() : s.finish(kDjCounters);
    };
    if constexpr (AN) {
        return by_width_enc(pk.width, probe);
    } else {  // (8-byte raw codes do not come here)
        if (pk.width == 1) return probe(std::integral_constant<int, 1>());
        if (pk.width == 2) return probe(std::integral_constant<int, 2>());
        return probe(std::integral_constant<int, 4>());
    }
}

size_t join_scratch(uint64_t nb, uint64_t np) {
    const uint64_t cap = ht_capacity(nb) + 1;
    const uint64_t nt = (np + kProbeTile - 1) / kProbeTile;
    return cap * (8 + 4 + 4 + 4 + 8 + 16) + 256 + nb * 8 + np * 4 + (scan_groups(cap) + 1) * 8 + nt * 12 +
           (scan_groups(nt) + 1) * 8 + 16 * 1024;
}

// Build on `bk` (nb rows), probe with `pk` (np rows); the output total lands
// in counter 0.  A sized call (`out` given) reads the total back once the matches
// are counted, gets its columns, and has the total in out->count.
int run_hash_join(OpScope& s, const KeyCfg& bk, uint64_t nb, const KeyCfg& pk, uint64_t np, JoinOut o, ahead_bat* out) {
    cudaStream_t st = s.ctx->stream;
    const uint32_t cap = ht_capacity(nb);
    HashTab h;
    h.mask = cap - 1;
    h.keys = (uint64_t*)s.alloc((size_t)(cap + 1) * 8);
    h.cnt = (uint32_t*)s.alloc((size_t)(cap + 1) * 4);
    h.off = (uint32_t*)s.alloc((size_t)(cap + 1) * 4);
    h.cur = (uint32_t*)s.alloc((size_t)(cap + 1) * 4);
    h.rows = (uint32_t*)s.alloc(nb * 4 + 4);
    uint32_t* slot_of = (uint32_t*)s.alloc(nb * 4 + 4);
    uint32_t* pslot = (uint32_t*)s.alloc(np * 4 + 4);
    cudaMemsetAsync(h.keys, 0xff, (size_t)(cap + 1) * 8, st);
    cudaMemsetAsync(h.cnt, 0, (size_t)(cap + 1) * 4, st);
    cudaMemsetAsync(h.cur, 0, (size_t)(cap + 1) * 4, st);
    const int g = s.ctx->num_sms * 8;
    ht_build_kernel<<<grid_for(nb, 256), 256, 0, st>>>(h, bk, nb, slot_of);
    // segment starts: scan of the slot counts (the compaction's two-level scan)
    CompactBufs sb;
    sb.words = nullptr;
    sb.counts = h.cnt;
    sb.offsets = (uint64_t*)s.alloc((size_t)(cap + 1) * 8);
    sb.gbase = (uint64_t*)s.alloc((size_t)scan_groups(cap + 1) * 8);
    sb.totals = s.d_counters + 60;
    sb.done = (uint32_t*)(s.d_counters + kScanDone);
    sb.ntiles = cap + 1;
    sb.nchan = 1;
    launch_scan(s, sb);
    ht_offsets_kernel<<<grid_for(cap + 1, 256), 256, 0, st>>>(h, sb);
    ht_fill_kernel<<<grid_for(nb, 256), 256, 0, st>>>(h, slot_of, nb);
    ht_order_kernel<<<grid_for(cap + 1, 256), 256, 0, st>>>(h, cap + 1);
    // single build rows go straight into the probe entries while rows fit 31 bits
    const bool direct = nb < (uint64_t)(kDirect - 1);
    ProbeSlot* pt = (ProbeSlot*)s.alloc((size_t)(cap + 1) * sizeof(ProbeSlot));
    ht_pack_kernel<<<grid_for(cap + 1, 256), 256, 0, st>>>(h, pt, cap + 1, direct);
    s.launched(5);
    const uint32_t nt = (uint32_t)((np + kProbeTile - 1) / kProbeTile);
    CompactBufs pb;
    pb.words = nullptr;
    pb.counts = (uint32_t*)s.alloc((size_t)nt * 4);
    pb.offsets = (uint64_t*)s.alloc((size_t)nt * 8);
    pb.gbase = (uint64_t*)s.alloc((size_t)scan_groups(nt) * 8);
    pb.totals = s.d_counters;
    pb.done = sb.done;
    pb.ntiles = nt;
    pb.nchan = 1;
    const uint32_t pg = nt < (uint32_t)g ? nt : (uint32_t)g;
    probe_count_kernel<<<pg, 256, 0, st>>>(pt, h.mask, direct, pk, np, pslot, pb);
    s.launched();
    launch_scan(s, pb);
    if (out) {
        const int rc = s.finish(1);
        if (rc) return rc;
        out->count = o.cap = s.counter(0);
        if (!s.take(&out->head, 0, o.cap) || !s.take(&out->tail, 1, o.cap))
            return fail(s.ctx, AHEAD_NO_MEMORY, "output allocation failed");
        o.oh = out->head.data;
        o.ot = out->tail.data;
    }
    probe_emit_kernel<<<pg, 256, 0, st>>>(pt, h.rows, np, pslot, pb, o);
    s.launched();
    return AHEAD_OK;
}

bool small_res(int t) { return t == AHEAD_RESTINY || t == AHEAD_RESSHORT || t == AHEAD_RESINT; }

KeyCfg key_cfg(const ahead_col& c, int dec, int keybase, int largerbase, bool cond) {
    KeyCfg k;
    k.col = dcol(c);
    k.width = type_width(c.type);
    k.dec = dec;
    k.ainv = c.Ainv & wmask(k.width);
    k.keymask = wmask(keybase);
    k.largermask = wmask(largerbase);
    k.condmax = cond ? wmask(keybase) : ~0ull;
    return k;
}

// ------------------------------------------------------ positional joins
// matchjoinAN<H1, resoid, void, T2> (matchjoinAN.tcc:271-298) and, with
// CHECKED = false, the unencoded matchjoin<H1, oid, void, T2>
// (Normal/matchjoin.tcc:140-157).  Streams: 0 kept, 1 bad head, 2 bad
// position, 3 corrupt fetched value.
template <bool CHECKED>
struct MjPosOp {
    static constexpr int W = CHECKED ? 8 : 4;
    static constexpr int NCH = CHECKED ? 4 : 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = true;
    static constexpr bool EMIT_V = true;
    static constexpr int NOUT = 2;
    const char* base;
    DCol h1c, t2c;
    uint64_t at1inv, ah1inv, ah1max, sz, fh, ft, cap, aoid, ec1, ec2, ec4;
    uint64_t *e1, *e2, *e4, *acc;
    void *oh, *ot;
    int ohw, otw, reenc, h1enc, t2enc;
    AHEAD_DEV uint64_t pos2(uint64_t v) const { return CHECKED ? v * at1inv : v; }
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t row, uint64_t&) const {
        uint32_t bits = 0;
        if (CHECKED && h1enc && load_at(h1c, row) * ah1inv > ah1max) bits |= 2u;
        const uint64_t p = pos2(v);
        if (p >= sz) return bits | (CHECKED ? 4u : 0u);
        if (CHECKED && t2enc && dec_if(t2c, load_at(t2c, p), t2c.ainv) > t2c.umax) return bits | 8u;
        return bits | 1u;
    }
    template <class V, int U>
    AHEAD_DEV void rows0(const V (&v)[U], uint64_t row0, const uint32_t (&idx)[U], uint64_t (&x)[2][U]) const {
        uint64_t p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = pos2(v[u]);
        gather_rows(t2c, p, x[1]);
        load_rows(h1c, row0, idx, x[0]);
        if (reenc) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                x[0][u] = dec_if(h1c, x[0][u], fh);
                x[1][u] = dec_if(t2c, x[1][u], ft);
            }
        }
    }
    AHEAD_DEV uint64_t cap0() const { return cap; }
    AHEAD_DEV void* optr(int k) const { return k == 0 ? oh : ot; }
    AHEAD_DEV int owidth(int k) const { return k == 0 ? ohw : otw; }
    AHEAD_DEV void emit(int c, uint64_t pos, uint64_t v, uint64_t row) const {
        if (c == 1) {
            if (pos < ec1) e1[pos] = row * aoid;
        } else if (c == 2) {
            if (pos < ec2) e2[pos] = row * aoid;
        } else if (c == 3) {
            if (pos < ec4) e4[pos] = pos2(v) * aoid;
        }
    }
};

// fetchjoinAN (matchjoinAN.tcc:330-351) and, with CHECKED = false, fetchjoin
// (Normal/matchjoin.tcc:159-178).  Streams: 0 kept, 1 bad OID, 2 corrupt value.
template <bool CHECKED>
struct FetchOp {
    static constexpr int W = CHECKED ? 8 : 4;
    static constexpr int NCH = CHECKED ? 3 : 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = true;
    static constexpr bool EMIT_V = true;
    static constexpr int NOUT = 1;
    const char* base;
    DCol t2c;
    uint64_t at1inv, at2inv, at2max, vsz, fac, cap, aoid, ec1, ec2;
    uint64_t *e1, *e2, *acc;
    void* ot;
    int otw, reenc, w2;
    AHEAD_DEV uint64_t pos(uint64_t v) const { return CHECKED ? v * at1inv : v; }
    AHEAD_DEV bool bad(uint64_t t2) const {
        // the check has no cast: 16-bit codes are multiplied as 32-bit ints
        if (w2 == 2) return (int32_t)(uint32_t)(t2 * at2inv) > (int32_t)at2max;
        return mulw(t2, at2inv, w2) > at2max;
    }
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t, uint64_t&) const {
        const uint64_t p = pos(v);
        if (p >= vsz) return CHECKED ? 2u : 0u;
        if (CHECKED && bad(load_at(t2c, p))) return 4u;
        return 1u;
    }
    template <class V, int U>
    AHEAD_DEV void rows0(const V (&v)[U], uint64_t, const uint32_t (&)[U], uint64_t (&x)[1][U]) const {
        uint64_t p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = pos(v[u]);
        gather_rows(t2c, p, x[0]);
        if (reenc) {
#pragma unroll
            for (int u = 0; u < U; ++u) x[0][u] = mulw(x[0][u], fac, w2);
        }
    }
    AHEAD_DEV uint64_t cap0() const { return cap; }
    AHEAD_DEV void* optr(int) const { return ot; }
    AHEAD_DEV int owidth(int) const { return otw; }
    AHEAD_DEV void emit(int c, uint64_t p, uint64_t v, uint64_t row) const {
        if (c == 1) {
            if (p < ec1) e1[p] = row * aoid;
        } else if (c == 2) {
            if (p < ec2) e2[p] = pos(v) * aoid;
        }
    }
};

// The positional joins in one pass: almost every row is kept, so row i's output
// goes to position i at once and the rows to drop are listed (see DropList).
// kRows rows per lane, their list entries, then their gathers in flight
// together.  What bounds it is the gather: at 12M OIDs of a fifth of a 60M-row
// 8-byte column nearly 60 % of the column's sectors are read (571 MB with the
// list and the outputs).  Warps stop once the list of dropped rows is over: with half
// of 30M OIDs past the column the pass took 162 us before the compaction's 116.
struct PosArgs {
    const char* base;   // the OID list's codes
    uint64_t n, inv, sz;
    DCol h1c, t2c;      // head of the list, fetched column
    uint64_t fh, ft;    // re-encoding factors
    void *oh, *ot;      // (oh null: fetchjoin, no head output)
    int ohw, otw, reenc, head_err, t2enc, w2;
    ErrList herr;       // corrupt heads
    DropList drops;     // kind 0: OID past the column, kind 1: corrupt value
};
constexpr int kPosRows = 4;

template <bool CHECKED, bool FETCH>
__global__ void __launch_bounds__(256) pos_join_kernel(PosArgs a) {
    constexpr int W = CHECKED ? 8 : 4;
    typedef typename std::conditional<W == 8, uint64_t, uint32_t>::type V;
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5, span = 32 * kPosRows;
    for (uint64_t r0 = warp * span; r0 < a.n; r0 += warps * span) {
        const uint32_t cnt = a.n - r0 < span ? (uint32_t)(a.n - r0) : (uint32_t)span;
        uint32_t idx[kPosRows];
        V v[kPosRows];
        uint64_t p[kPosRows], val[2][kPosRows];
        bool ok[kPosRows], over = false;
#pragma unroll
        for (int u = 0; u < kPosRows; ++u) {
            idx[u] = lane + 32 * u < cnt ? lane + 32 * u : 0;
            v[u] = gmem_ld<W>(a.base + r0 * W, idx[u]);
        }
#pragma unroll
        for (int u = 0; u < kPosRows; ++u) {
            p[u] = CHECKED ? v[u] * a.inv : v[u];
            ok[u] = p[u] < a.sz;
            if (!ok[u]) {
                if (lane + 32 * u < cnt) over |= a.drops.add(r0 + idx[u], 0);
                p[u] = 0;  // (the column has a row: sz > 0)
            }
        }
        if (__any_sync(kFull, over)) return;
        gather_rows(a.t2c, p, val[1]);
        if (!FETCH) {
            if (CHECKED && a.h1c.type != AHEAD_VOID && a.h1c.data == a.base) {  // a mirrored list: the head is the OID itself
#pragma unroll
                for (int u = 0; u < kPosRows; ++u) val[0][u] = v[u];
            } else {
                load_rows(a.h1c, r0, idx, val[0]);
            }
            if (CHECKED && a.head_err) {
#pragma unroll
                for (int u = 0; u < kPosRows; ++u)
                    if (val[0][u] * a.h1c.ainv > a.h1c.umax && lane + 32 * u < cnt) a.herr.add(r0 + idx[u]);
            }
        }
        if (CHECKED && a.t2enc) {
#pragma unroll
            for (int u = 0; u < kPosRows; ++u) {
                // fetchjoinAN's check has no cast: 16-bit codes are multiplied as 32-bit ints
                const bool bad = FETCH && a.w2 == 2
                                     ? (int32_t)(uint32_t)(val[1][u] * a.t2c.ainv) > (int32_t)a.t2c.umax
                                     : mulw(val[1][u], a.t2c.ainv, a.w2) > a.t2c.umax;
                if (bad && ok[u] && lane + 32 * u < cnt) over |= a.drops.add(r0 + idx[u], 1);
            }
            if (__any_sync(kFull, over)) return;
        }
        if (a.reenc) {
#pragma unroll
            for (int u = 0; u < kPosRows; ++u) {
                if (!FETCH) val[0][u] = dec_if(a.h1c, val[0][u], a.fh);
                val[1][u] = dec_if(a.t2c, val[1][u], a.ft);
            }
        }
        auto store = [&](void* o, int w, const uint64_t (&x)[kPosRows]) {
            auto st = [&](auto* q) {
                q += r0 + lane;
#pragma unroll
                for (int u = 0; u < kPosRows; ++u)
                    if (lane + 32 * u < cnt) q[32 * u] = x[u];
            };
            if (w == 8) st((uint64_t*)o);
            else if (w == 4) st((uint32_t*)o);
            else if (w == 2) st((uint16_t*)o);
            else st((uint8_t*)o);
        };
        if (!FETCH) store(a.oh, a.ohw, val[0]);
        store(a.ot, a.otw, val[1]);
    }
}

// Where the one-pass form pays and applies: more rows than one block's
// compaction takes (8,192), room for every row, and a column to fetch from.
inline bool pos_one_pass(uint64_t n, uint64_t cap, uint64_t sz) {
    return n > 32 * short_k(8) * (uint64_t)kOneBlockTiles && n <= cap && sz > 0;
}

constexpr int kPosHead = 30, kPosDrops = 31, kPosCounters = 33;  // counters

// Runs the one-pass form; *kept = rows kept.  Returns AHEAD_UNSUPPORTED when
// too many rows are dropped, or the device memory is short, and the compaction
// has to run.  `dense_head`: every
// head is known to read as corrupt, so its vector is made by a column check.
template <bool CHECKED, bool FETCH>
int run_pos_join(OpScope& s, PosArgs& a, const ahead_col* head, uint64_t aoid, bool dense_head, ahead_errvec* eh,
                 ahead_errvec* e0, ahead_errvec* e1, uint64_t* kept) {
    if (((uintptr_t)a.oh | (uintptr_t)a.ot) & 3) return AHEAD_UNSUPPORTED;  // (narrow gaps are closed by words)
    const uint64_t n = a.n;
    const bool want_head = a.head_err && eh;
    const size_t check = want_head ? colcheck_scratch(n) : 0;
    int rc = s.reserve(drop_scratch(n, (FETCH ? 0 : a.ohw) + a.otw) + kErrListBytes + check);
    if (rc) return rc == AHEAD_NO_MEMORY ? AHEAD_UNSUPPORTED : rc;  // (the compaction needs a tenth of it)
    a.herr = err_list(s, kPosHead);
    a.drops = drop_list(s, kPosDrops);
    uint64_t* sorted = (uint64_t*)s.alloc(kMaxDrops * 8);
    if (dense_head) a.head_err = 0;
    const uint64_t blocks = (n + 256 * kPosRows - 1) / (256 * kPosRows);
    const uint32_t most = (uint32_t)s.ctx->num_sms * 32;
    pos_join_kernel<CHECKED, FETCH><<<blocks < most ? (uint32_t)blocks : most, 256, 0, s.ctx->stream>>>(a);
    s.launched();
    auto check_head = [&] { run_colcheck(s, *head, n, a.h1c.ainv, a.h1c.umax, 8, aoid, eh, 1); };
    if (want_head && dense_head) check_head();
    rc = s.finish(kPosCounters);
    if (rc) return rc;
    const uint64_t k = s.counter(kPosDrops), k1 = s.counter(kPosDrops + 1);
    if (!shift_fits(s, n, k, (FETCH ? 0 : a.ohw) + a.otw)) return AHEAD_UNSUPPORTED;
    *kept = n - k;
    if (e0) e0->count = k - k1;
    if (e1) e1->count = k1;
    if (want_head && dense_head) eh->count = s.counter(1);
    if (k) {
        sort_drops_kernel<<<1, 1024, 0, s.ctx->stream>>>(a.drops.rows, (uint32_t)k, sorted, (const uint64_t*)a.base,
                                                         a.inv, aoid, edata(e0), ecap(e0), edata(e1), ecap(e1));
        s.launched();
        if (FETCH) launch_shift(s, n, sorted, (uint32_t)k, a.ot, a.otw);
        else launch_shift(s, n, sorted, (uint32_t)k, a.ot, a.otw, a.oh, a.ohw);
    }
    if (want_head && !dense_head && !settle_err_list(s, a.herr, kPosHead, aoid, eh)) {
        // (the gaps' edges may have taken the scratch up to its end: the check, behind
        // them in the stream, starts over in it)
        rc = s.reserve(check);
        if (rc) return rc;
        check_head();
        rc = s.finish(2);
        if (rc) return rc;
        eh->count = s.counter(1);
    }
    return s.wait();
}

// ------------------------------------------------------------ merge joins
struct MergeSide {
    DCol key, other;  // key column (decoded when encoded) and the other column
    int key_enc, other_enc;
};

AHEAD_DEV uint64_t key_val(const DCol& c, uint64_t row) { return dec_if(c, load_at(c, row), c.ainv); }

// Flags (bit 0) a key that does not strictly increase -- the parallel merge
// is exact only without one -- and (bit 1) any corrupt value in either column,
// which decides whether error positions must be produced.  Both inputs in one
// launch (blockIdx.y), 256 rows per warp and step, eight loads in flight per
// lane; the key before a lane's comes from its neighbour.
__global__ void __launch_bounds__(256) merge_check_kernel(MergeSide ma, uint64_t na, MergeSide mb, uint64_t nb,
                                                          uint32_t* flag) {
    constexpr int U = 8;
    const MergeSide m = blockIdx.y ? mb : ma;
    const uint64_t n = blockIdx.y ? nb : na;
    // (a mirrored list is checked once)
    const bool other = m.other_enc && !(m.key_enc && m.other.data == m.key.data && m.other.ainv == m.key.ainv &&
                                        m.other.umax == m.key.umax);
    const int lane = threadIdx.x & 31;
    uint32_t f = 0;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r0 = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * (32 * U); r0 < n;
         r0 += warps * (32 * U)) {
        const uint32_t cnt = n - r0 < 32 * U ? (uint32_t)(n - r0) : 32 * U;
        uint32_t idx[U];
        uint64_t k[U];
#pragma unroll
        for (int q = 0; q < U; ++q) idx[q] = lane + 32 * q < cnt ? lane + 32 * q : 0;
        load_rows(m.key, r0, idx, k);
        uint64_t last = r0 ? dec_if(m.key, load_at(m.key, r0 - 1), m.key.ainv) : 0;
#pragma unroll
        for (int q = 0; q < U; ++q) {
            k[q] = dec_if(m.key, k[q], m.key.ainv);
            const uint64_t up = __shfl_up_sync(kFull, k[q], 1);
            const uint64_t before = lane ? up : last;
            last = __shfl_sync(kFull, k[q], 31);
            if (lane + 32 * q < cnt) {
                if (r0 + lane + 32 * q && before >= k[q]) f |= 1u;
                if (m.key_enc && k[q] > m.key.umax) f |= 2u;
            }
        }
        if (other) {
            load_rows(m.other, r0, idx, k);
#pragma unroll
            for (int q = 0; q < U; ++q)
                if (dec_if(m.other, k[q], m.other.ainv) > m.other.umax) f |= 2u;
        }
    }
    f = __reduce_or_sync(kFull, f);
    if (f && lane == 0) atomicOr(flag, f);
}

// Error positions of the reference's merge loop (matchjoinAN.tcc:101-136) for
// two strictly increasing key sequences, derived per row instead of by running
// the loop.  Walking the loop over the merged order of the keys shows:
//  - a first-input row is checked once, when the inner p1 loop passes it:
//    exactly when it is unmatched and some second-input key is larger
//    (matched rows are emitted unchecked);
//  - a second-input row j is checked at the top of an outer iteration when
//    j == 0, row j-1 matched, or a first-input key lies strictly between keys
//    j-1 and j; an unmatched row is checked again when the inner p2 loop
//    passes it, which happens when a larger first-input key exists; without
//    one, only the first unmatched row after the last first-input key is
//    checked (once), and only when that last key is itself unmatched (a match
//    of the last first-input key ends the loop).
// Each check pushes `row * AOID` into the vector of each corrupt column.
struct MergeErrs {
    DCol h1, t1, h2, t2;
    uint64_t n1, n2, aoid;
    int eh1, et1, eh2, et2;
    const uint64_t* l1m;      // device word: the last first-input key occurs in the second input
    AHEAD_DEV uint64_t lb1(uint64_t x) const {  // first-input keys below x
        uint64_t lo = 0, hi = n1;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (key_val(t1, mid) < x) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    }
    AHEAD_DEV bool in2(uint64_t k) const {
        uint64_t lo = 0, hi = n2;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (key_val(h2, mid) < k) lo = mid + 1;
            else hi = mid;
        }
        return lo < n2 && key_val(h2, lo) == k;
    }
    // checks of row r of `side` (0: first input, 1: second) and which of its
    // two columns are corrupt
    AHEAD_DEV uint32_t checks(int side, uint64_t r, bool& bad_a, bool& bad_b) const {
        if (side == 0) {
            const uint64_t k = key_val(t1, r);
            bad_a = eh1 && key_val(h1, r) > h1.umax;
            bad_b = et1 && k > t1.umax;
            if (!(bad_a || bad_b)) return 0;
            return (k < key_val(h2, n2 - 1) && !in2(k)) ? 1u : 0u;
        }
        const uint64_t K = key_val(h2, r);
        bad_a = eh2 && K > h2.umax;
        bad_b = et2 && key_val(t2, r) > t2.umax;
        if (!(bad_a || bad_b)) return 0;
        const uint64_t L = lb1(K);
        const bool matched = L < n1 && key_val(t1, L) == K;
        bool top = r == 0;
        uint64_t upto_prev = 0;  // first-input keys <= key r-1
        if (r > 0) {
            const uint64_t Kp = key_val(h2, r - 1);
            const uint64_t Lp = lb1(Kp);
            const bool mp = Lp < n1 && key_val(t1, Lp) == Kp;
            upto_prev = Lp + (mp ? 1 : 0);
            top = mp || L > upto_prev;
        }
        if (matched) return top ? 1u : 0u;
        if (L < n1) return (top ? 1u : 0u) + 1u;
        return ((r == 0 || upto_prev < n1) && !*l1m) ? 1u : 0u;
    }
};

constexpr int kMeRows = 16;
constexpr int kMeThreads = 256;
constexpr int kMeTile = kMeRows * kMeThreads;

__global__ void merge_last_kernel(MergeErrs m, uint64_t* out) { out[0] = m.in2(key_val(m.t1, m.n1 - 1)) ? 1 : 0; }

// Exclusive scan of two counters over a block of kMeThreads threads.
AHEAD_DEV void block_scan2(uint32_t& a, uint32_t& b, uint32_t* tot_a, uint32_t* tot_b) {
    __shared__ uint32_t s_a[kMeThreads / 32], s_b[kMeThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t ia = warp_incl_scan(a), ib = warp_incl_scan(b);
    if (lane == 31) {
        s_a[wid] = ia;
        s_b[wid] = ib;
    }
    __syncthreads();
    uint32_t pa = 0, pb = 0, ta = 0, tb = 0;
    for (int w = 0; w < kMeThreads / 32; ++w) {
        if (w < wid) {
            pa += s_a[w];
            pb += s_b[w];
        }
        ta += s_a[w];
        tb += s_b[w];
    }
    a = pa + ia - a;
    b = pb + ib - b;
    *tot_a = ta;
    *tot_b = tb;
    __syncthreads();
}

__global__ void __launch_bounds__(kMeThreads) merge_err_count_kernel(MergeErrs m, int side, uint64_t n,
                                                                     uint32_t* tcount) {
    const uint64_t t0 = (uint64_t)blockIdx.x * kMeTile;
    uint32_t ca = 0, cb = 0;
    for (int k = 0; k < kMeRows; ++k) {
        const uint64_t r = t0 + (uint64_t)threadIdx.x * kMeRows + k;
        if (r >= n) break;
        bool ba, bb;
        const uint32_t c = m.checks(side, r, ba, bb);
        ca += ba ? c : 0;
        cb += bb ? c : 0;
    }
    uint32_t ta, tb;
    block_scan2(ca, cb, &ta, &tb);
    if (threadIdx.x == 0) {
        tcount[2 * blockIdx.x] = ta;
        tcount[2 * blockIdx.x + 1] = tb;
    }
}

// One block: exclusive offsets of the tile counts; totals into tot[0], tot[1].
__global__ void __launch_bounds__(kMeThreads) merge_err_scan_kernel(const uint32_t* tcount, uint64_t* toff,
                                                                    uint32_t ntiles, uint64_t* tot) {
    __shared__ uint64_t s_base[2];
    if (threadIdx.x == 0) s_base[0] = s_base[1] = 0;
    __syncthreads();
    for (uint32_t c0 = 0; c0 < ntiles; c0 += kMeThreads) {
        const uint32_t t = c0 + threadIdx.x;
        uint32_t a = t < ntiles ? tcount[2 * t] : 0, b = t < ntiles ? tcount[2 * t + 1] : 0;
        uint32_t ta, tb;
        block_scan2(a, b, &ta, &tb);
        if (t < ntiles) {
            toff[2 * t] = s_base[0] + a;
            toff[2 * t + 1] = s_base[1] + b;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_base[0] += ta;
            s_base[1] += tb;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        tot[0] = s_base[0];
        tot[1] = s_base[1];
    }
}

__global__ void __launch_bounds__(kMeThreads) merge_err_write_kernel(MergeErrs m, int side, uint64_t n,
                                                                     const uint64_t* toff, uint64_t* ea,
                                                                     uint64_t capa, uint64_t* eb, uint64_t capb) {
    const uint64_t t0 = (uint64_t)blockIdx.x * kMeTile;
    uint32_t ca = 0, cb = 0;
    uint32_t mult[kMeRows];
    uint32_t bad[kMeRows];
    for (int k = 0; k < kMeRows; ++k) {
        const uint64_t r = t0 + (uint64_t)threadIdx.x * kMeRows + k;
        mult[k] = 0;
        bad[k] = 0;
        if (r < n) {
            bool ba, bb;
            mult[k] = m.checks(side, r, ba, bb);
            bad[k] = (ba ? 1u : 0u) | (bb ? 2u : 0u);
            ca += ba ? mult[k] : 0;
            cb += bb ? mult[k] : 0;
        }
    }
    uint32_t ta, tb;
    block_scan2(ca, cb, &ta, &tb);
    uint64_t pa = toff[2 * blockIdx.x] + ca, pb = toff[2 * blockIdx.x + 1] + cb;
    for (int k = 0; k < kMeRows; ++k) {
        const uint64_t r = t0 + (uint64_t)threadIdx.x * kMeRows + k;
        for (uint32_t c = 0; c < mult[k]; ++c) {
            if (bad[k] & 1u) {
                if (ea && pa < capa) ea[pa] = r * m.aoid;
                ++pa;
            }
            if (bad[k] & 2u) {
                if (eb && pb < capb) eb[pb] = r * m.aoid;
                ++pb;
            }
        }
    }
}

// Intersection of two strictly increasing key sequences: each tile of the
// first input only meets the second input's keys from its own first key to the
// next tile's, a stretch that merge_part_kernel finds for all tiles at once;
// each row then searches its tile's stretch (a few hundred keys, in L1).  No
// structure over the whole key range is built, so the range's width does not
// matter.  While a tile's keys span at most kMergeMap values (selections of
// ordinary shares do), the stretch marks a byte map of that span in shared
// memory and a row's search is one byte; a wider tile searches its stretch.
// When the second input's tail is its head (a mirrored selection), the matched
// value is the key itself and the emit pass does not search at all.
// At 29M and 16M plain 4-byte OIDs of 60M, a binary search over all of the
// second input per row took 775 us to classify and 285 us to emit, a search of
// the stretch 234 and 170; this takes 57 and 54 (180 MB read per pass), and 18 us for
// the stretches.
struct MergeParts {
    DCol k1, k2;  // key columns
    uint64_t n1, n2;
    uint64_t* part;  // [tiles + 1] first row of the second input at or past each tile's first key
};
constexpr uint64_t kMergeTile = 32 * short_k(8);  // rows per tile (driving columns of 2, 4 or 8 bytes)
constexpr uint32_t kMergeMap = 4096;

__global__ void __launch_bounds__(256) merge_part_kernel(MergeParts m, uint32_t tiles) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > tiles) return;
    uint64_t lo = 0, hi = m.n2;
    if (t == tiles) {
        lo = hi;
    } else {
        const uint64_t k = key_val(m.k1, (uint64_t)t * kMergeTile);
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (key_val(m.k2, mid) < k) lo = mid + 1;
            else hi = mid;
        }
    }
    m.part[t] = lo;
}

template <int WW>
struct IsectOp {
    static constexpr int W = WW;
    static constexpr int NCH = 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = true;
    static constexpr bool EMIT_V = false;
    static constexpr int NOUT = 2;
    const char* base;
    DCol t1c, h1c, h2c, t2c;
    uint64_t fh, ft, cap;
    uint64_t* acc;
    void *oh, *ot;
    int ohw, otw, reenc;
    int mirror2;   // the second input's tail is its head: its value is key * a2
    uint64_t a2;
    const uint64_t* part;
    const uint32_t* flag;  // merge_check_kernel's
    uint64_t lo, len;  // the tile's stretch of the second input
    // Keys out of order have stretches that start behind their end, and a search
    // that misses a marked key: then no tile has a stretch, so that nothing is
    // searched, kept or gathered, and the replayed loop makes the result.
    AHEAD_DEV void tile(uint32_t t) {
        lo = __ldg((const unsigned long long*)part + t);
        len = (__ldg(flag) & 1u) ? 0 : __ldg((const unsigned long long*)part + t + 1) - lo;
    }
    AHEAD_DEV uint64_t find(uint64_t row) const {  // ~0: no match
        const uint64_t k = key_val(t1c, row);
        uint64_t at = lo, m = len;
        while (m >> 32) {  // (a stretch of 2^32 rows and more)
            const uint64_t half = m >> 1;
            if (key_val(h2c, at + half) < k) {
                at += half + 1;
                m -= half + 1;
            } else {
                m = half;
            }
        }
        uint32_t a = 0, b = (uint32_t)m;
        while (a < b) {
            const uint32_t mid = a + (b - a) / 2;
            if (key_val(h2c, at + mid) < k) a = mid + 1;
            else b = mid;
        }
        at += a;
        return (at < lo + len && key_val(h2c, at) == k) ? at : ~0ull;
    }
    AHEAD_DEV uint32_t eval(uint64_t, uint64_t row, uint64_t&) const { return find(row) != ~0ull ? 1u : 0u; }
    template <class V, int U>
    AHEAD_DEV void rows0(const V (&)[U], uint64_t row0, const uint32_t (&idx)[U], uint64_t (&x)[2][U]) const {
        load_rows(h1c, row0, idx, x[0]);
        if (mirror2) {
            load_rows(t1c, row0, idx, x[1]);
#pragma unroll
            for (int u = 0; u < U; ++u) x[1][u] = dec_if(t1c, x[1][u], t1c.ainv) * a2;
        } else {
            uint64_t p[U];
#pragma unroll
            for (int u = 0; u < U; ++u) p[u] = find(row0 + idx[u]);
            gather_rows(t2c, p, x[1]);
        }
        if (reenc) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                x[0][u] = dec_if(h1c, x[0][u], fh);
                x[1][u] = dec_if(t2c, x[1][u], ft);
            }
        }
    }
    AHEAD_DEV uint64_t cap0() const { return cap; }
    AHEAD_DEV void* optr(int k) const { return k == 0 ? oh : ot; }
    AHEAD_DEV int owidth(int k) const { return k == 0 ? ohw : otw; }
};

// Pass 1 through the byte map, one warp per tile; word s of a tile is the
// ballot of its rows 32 s ... 32 s + 31.
template <class Op>
__global__ void __launch_bounds__(kCThreads) merge_classify_kernel(Op op, uint64_t n, CompactBufs cb) {
    constexpr int K = short_k(8);
    __shared__ __align__(16) uint8_t s_map[kCWarps][kMergeMap];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* map = s_map[warp];
    const uint32_t tile = blockIdx.x * kCWarps + warp;
    if (tile >= cb.ntiles) return;
    op.tile(tile);
    const uint64_t row0 = (uint64_t)tile * kMergeTile;
    const uint32_t m = n - row0 < kMergeTile ? (uint32_t)(n - row0) : (uint32_t)kMergeTile;
    uint32_t idx[K];
    uint64_t k[K];
#pragma unroll
    for (int s = 0; s < K; ++s) idx[s] = lane + 32 * s < m ? lane + 32 * s : m - 1;
    load_rows(op.t1c, row0, idx, k);
#pragma unroll
    for (int s = 0; s < K; ++s) k[s] = dec_if(op.t1c, k[s], op.t1c.ainv);
    const uint64_t first = __shfl_sync(kFull, k[0], 0), last = __shfl_sync(kFull, k[K - 1], 31);
    const uint64_t span = last - first + 1;
    uint32_t word = 0;
    if (span && span <= kMergeMap && op.len <= kMergeMap) {
        const uint32_t w = (uint32_t)span, len = (uint32_t)op.len;
        for (uint32_t i = lane; i < (w + 15) / 16; i += 32) reinterpret_cast<uint4*>(map)[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        for (uint32_t j0 = lane; j0 < len; j0 += 128) {
            uint32_t at[4];
            uint64_t x[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) at[q] = j0 + 32 * q < len ? j0 + 32 * q : j0;
            load_rows(op.h2c, op.lo, at, x);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t d = dec_if(op.h2c, x[q], op.h2c.ainv) - first;
                if (d < w) map[d] = 1;
            }
        }
        __syncwarp();
#pragma unroll
        for (int s = 0; s < K; ++s) {
            const uint64_t d = k[s] - first;
            const uint32_t b = __ballot_sync(kFull, lane + 32 * s < m && d < w && map[d < w ? d : 0]);
            if (lane == s) word = b;
        }
    } else {
#pragma unroll 1
        for (int s = 0; s < K; ++s) {
            const uint64_t row = row0 + lane + 32 * s;
            const uint32_t b = __ballot_sync(kFull, lane + 32 * s < m && op.find(row) != ~0ull);
            if (lane == s) word = b;
        }
    }
    if (lane < K) cb.words[(size_t)tile * K + lane] = word;
    const uint32_t count = __reduce_add_sync(kFull, (uint32_t)__popc(word));
    if (lane == 0) cb.counts[tile] = count;
}

size_t merge_scratch(uint64_t n1) {
    return compact_scratch<IsectOp<8>>(n1) + (n1 / kMergeTile + 2) * 8 + 1024;
}

// The checks (flag in counter kMergeFlag) and the intersection (total in
// counter 0), both read back; the intersection counts only when the flag's bit 0
// stays clear.  `dw`: the
// driving column's width, at least 2.
constexpr int kMergeFlag = 40, kMergeCounters = 41;

int run_merge(OpScope& s, const DCol& t1, const DCol& h1, const DCol& h2, const DCol& t2, uint64_t n1, uint64_t n2,
              bool checked, int dw, int reenc, uint64_t fh, uint64_t ft, ahead_bat* out, uint64_t cap) {
    cudaStream_t st = s.ctx->stream;
    MergeSide ma{t1, h1, checked && t1.enc, checked && h1.enc};
    MergeSide mb{h2, t2, checked && h2.enc, checked && t2.enc};
    const uint64_t most = (n1 > n2 ? n1 : n2) / 4 + 1;
    const uint32_t cg = grid_for(most, 256), cl = (uint32_t)s.ctx->num_sms * 8;
    merge_check_kernel<<<dim3(cg < cl ? cg : cl, 2), 256, 0, st>>>(ma, n1, mb, n2,
                                                                   (uint32_t*)(s.d_counters + kMergeFlag));
    const uint32_t tiles = (uint32_t)((n1 + kMergeTile - 1) / kMergeTile);
    MergeParts mp{t1, h2, n1, n2, (uint64_t*)s.alloc(((size_t)tiles + 1) * 8)};
    merge_part_kernel<<<(tiles + 256) / 256, 256, 0, st>>>(mp, tiles);
    s.launched(2);
    const bool sized = s.sized(out, cap);
    return by_width_enc(dw, [&](auto tag) -> int {
        IsectOp<decltype(tag)::value> op;
        op.base = (const char*)(t1.type == AHEAD_VOID ? h1.data : t1.data);
        op.t1c = t1;
        op.h1c = h1;
        op.h2c = h2;
        op.t2c = t2;
        op.fh = fh;
        op.ft = ft;
        op.cap = (out->head.data && out->tail.data) ? cap : 0;
        op.acc = nullptr;
        op.oh = out->head.data;
        op.ot = out->tail.data;
        op.ohw = type_width(out->head.type);
        op.otw = type_width(out->tail.type);
        op.reenc = reenc;
        op.mirror2 = t2.type != AHEAD_VOID && t2.data == h2.data && t2.type == h2.type && t2.ainv == h2.ainv;
        op.a2 = h2.enc ? inv_pow2(h2.ainv, 64) : 1;
        op.part = mp.part;
        op.flag = (const uint32_t*)(s.d_counters + kMergeFlag);
        op.lo = op.len = 0;
        if (tiles <= kOneBlockTiles && !sized) {
            run_compact(s, op, n1, 0);
            return s.finish(kMergeCounters);
        }
        const CompactBufs cb = s.compact_bufs(n1, tiles, 1, 0);
        merge_classify_kernel<<<(tiles + kCWarps - 1) / kCWarps, kCThreads, 0, st>>>(op, n1, cb);
        s.launched();
        launch_scan(s, cb);
        if (sized) {
            int rc = s.finish(kMergeCounters);
            if (rc || (s.counter(kMergeFlag) & 1u)) return rc;
            op.cap = s.counter(0);
            if (!s.take(&out->head, 0, op.cap) || !s.take(&out->tail, 1, op.cap))
                return fail(s.ctx, AHEAD_NO_MEMORY, "output allocation failed");
            op.oh = out->head.data;
            op.ot = out->tail.data;
        }
        launch_emit(s, op, n1, cb);
        return sized ? s.wait() : s.finish(kMergeCounters);
    });
}

struct MergeSeq {
    DCol h1, t1, h2, t2;
    uint64_t n1, n2, fh, ft, aoid, cap;
    uint64_t ecap[4];
    uint64_t* e[4];
    void *oh, *ot;
    int ohw, otw, reenc, checked;
};

// The reference's merge loop (matchjoinAN.tcc:101-136, Normal/matchjoin.tcc:
// 49-72), one thread, for inputs that are not strictly increasing and clean.
// Counters: [0] output rows, [1..4] error counts.
__global__ void merge_seq_kernel(MergeSeq m, uint64_t* counters) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    uint64_t nout = 0, ne[4] = {0, 0, 0, 0};
    auto push = [&](int v, uint64_t pos) {
        if (!m.checked || !m.e[v]) {
            ++ne[v];
            return;
        }
        if (ne[v] < m.ecap[v]) m.e[v][ne[v]] = pos * m.aoid;
        ++ne[v];
    };
    const bool eh1 = m.checked && m.h1.enc, et1 = m.checked && m.t1.enc, eh2 = m.checked && m.h2.enc,
               et2 = m.checked && m.t2.enc;
    uint64_t p1 = 0, p2 = 0;
    while (p1 < m.n1 && p2 < m.n2) {
        uint64_t h2 = key_val(m.h2, p2);
        if (eh2 && h2 > m.h2.umax) push(2, p2);
        if (et2 && key_val(m.t2, p2) > m.t2.umax) push(3, p2);
        uint64_t t1 = key_val(m.t1, p1);
        bool valid;
        while ((valid = p1 < m.n1) && t1 < h2) {
            if (eh1 && key_val(m.h1, p1) > m.h1.umax) push(0, p1);
            if (et1 && t1 > m.t1.umax) push(1, p1);
            ++p1;
            if (p1 < m.n1) t1 = key_val(m.t1, p1);
        }
        if (valid) {
            while ((valid = p2 < m.n2) && t1 > h2) {
                if (eh2 && h2 > m.h2.umax) push(2, p2);
                if (et2 && key_val(m.t2, p2) > m.t2.umax) push(3, p2);
                ++p2;
                if (p2 < m.n2) h2 = key_val(m.h2, p2);
            }
            if (valid && t1 == h2) {
                if (nout < m.cap) {
                    uint64_t hv = load_at(m.h1, p1), tv = load_at(m.t2, p2);
                    if (m.reenc) {
                        hv = dec_if(m.h1, hv, m.fh);
                        tv = dec_if(m.t2, tv, m.ft);
                    }
                    store_at(m.oh, m.ohw, nout, hv);
                    store_at(m.ot, m.otw, nout, tv);
                }
                ++nout;
                ++p1;
                ++p2;
            }
        }
    }
    counters[0] = nout;
    for (int v = 0; v < 4; ++v) counters[1 + v] = ne[v];
}

// A sized call's columns for the replayed loop: each row it keeps takes one of
// either input, so the shorter one's length always fits, and a count of them
// would be the whole loop run twice.
int seq_columns(OpScope& s, ahead_bat* out, uint64_t n1, uint64_t n2, uint64_t& cap) {
    if (!s.sized(out, cap)) return AHEAD_OK;
    cap = n1 < n2 ? n1 : n2;
    if (!s.take(&out->head, 0, cap) || !s.take(&out->tail, 1, cap))
        return fail(s.ctx, AHEAD_NO_MEMORY, "output allocation failed");
    return AHEAD_OK;
}

__global__ void zip_kernel(DCol h1, DCol t2, uint64_t p1, uint64_t p2, uint64_t m, int reenc, uint64_t fh, uint64_t ft,
                           void* oh, int ohw, void* ot, int otw, uint64_t cap) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m && i < cap;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t hv = load_at(h1, p1 + i), tv = load_at(t2, p2 + i);
        if (reenc) {
            hv = dec_if(h1, hv, fh);
            tv = dec_if(t2, tv, ft);
        }
        store_at(oh, ohw, i, hv);
        store_at(ot, otw, i, tv);
    }
}

// Leading rows skipped before the zip of a void-void positional join
// (matchjoinAN.tcc:185-196): rows whose dense OID (mod 2^32) lies below the
// other side's seqbase.
uint64_t vv_skip(uint64_t my_seq, uint64_t other_seq, uint64_t n) {
    if (other_seq >= (1ull << 32)) return n;
    const uint64_t s0 = my_seq & 0xffffffffull;
    if (s0 >= other_seq) return 0;
    const uint64_t k = other_seq - s0;
    return k < n ? k : n;
}

struct CommonMj {
    int H1, T1, H2, T2;
};

void set_errs_present(ahead_errvec* errs, int p0, int p1, int p2, int p3) {
    if (!errs) return;
    ev_begin(&errs[0], p0);
    ev_begin(&errs[1], p1);
    ev_begin(&errs[2], p2);
    ev_begin(&errs[3], p3);
}

ahead_errvec* ev(ahead_errvec* errs, int k) { return errs ? &errs[k] : nullptr; }

// The string hash join's second step: copy each emitted row's matched
// right slot, and decode the left head where the reference emits it decoded.
__global__ void __launch_bounds__(256) str_gather_kernel(const uint32_t* rows, uint64_t n, const char* strs,
                                                         uint64_t width, char* out, bool decode, uint64_t ainv,
                                                         void* head, int hw) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const char* src = strs + (uint64_t)rows[i] * width;
        char* dst = out + i * width;
        for (uint64_t k = 0; k < width; ++k) dst[k] = src[k];
        if (decode) {
            if (hw == 8) ((uint64_t*)head)[i] *= ainv;
            else ((uint32_t*)head)[i] *= (uint32_t)ainv;
        }
    }
}

// fetchjoinAN with a string tail (FetchjoinAN<v2_str_t, false>,
// matchjoinAN.tcc:304-354): stream 0 = the rows whose OID is inside the
// column, written as their source row (the slots are gathered afterwards);
// stream 1 = the rest, reported as row * AOID.  The string tail is not
// encoded, so nothing else is checked.
struct FetchStrOp {
    static constexpr int W = 8;
    static constexpr int NCH = 2;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = false;
    static constexpr bool EMIT_V = true;
    static constexpr int NOUT = 1;
    const char* base;
    uint64_t ainv, count, aoid, cap, errcap;
    uint32_t* rows;
    uint64_t* err;
    uint64_t* acc;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t, uint64_t&) const { return v * ainv < count ? 1u : 2u; }
    AHEAD_DEV uint64_t out0(int, uint64_t v, uint64_t) const { return v * ainv; }
    AHEAD_DEV uint64_t cap0() const { return cap; }
    AHEAD_DEV void* optr(int) const { return rows; }
    AHEAD_DEV int owidth(int) const { return 4; }
    AHEAD_DEV void emit(int, uint64_t pos, uint64_t, uint64_t row) const {
        if (pos < errcap) err[pos] = row * aoid;
    }
};

// fetchjoin over a string tail (Normal/matchjoin.tcc:144-160): the rows whose
// oid_t is inside the column, as their source row; no checks.
struct FetchStrPlainOp {
    static constexpr int W = 4;
    static constexpr int NCH = 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = false;
    static constexpr bool EMIT_V = true;
    static constexpr int NOUT = 1;
    const char* base;
    uint64_t count, cap;
    uint32_t* rows;
    uint64_t* acc;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t, uint64_t&) const { return v < count ? 1u : 0u; }
    AHEAD_DEV uint64_t out0(int, uint64_t v, uint64_t) const { return v; }
    AHEAD_DEV uint64_t cap0() const { return cap; }
    AHEAD_DEV void* optr(int) const { return rows; }
    AHEAD_DEV int owidth(int) const { return 4; }
};

// The slots of a compacted row list, into `out` (the second step of both string fetch-joins).
int gather_str_rows(ahead_ctx* ctx, const uint32_t* rows, uint64_t n, const char* strs, uint64_t width, char* out) {
    if (!n || !out) return AHEAD_OK;
    str_gather_kernel<<<grid_for(n, 256), 256, 0, ctx->stream>>>(rows, n, strs, width, out, false, 0, nullptr, 8);
    ctx->launches += 1;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "kernel launch");
    e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? AHEAD_OK : cuda_fail(ctx, e, "cudaStreamSynchronize");
}

}  // namespace

namespace ahead {
int restiny_promoted_check(ahead_ctx* ctx, const uint16_t* codes, uint64_t n, uint32_t ainv, uint32_t umax,
                           uint64_t aoid, ahead_errvec* err);
}

extern "C" {

int ahead_gpu_hashjoin_str_an(ahead_ctx* ctx, const ahead_bat* l, const ahead_bat* r, const char* r_strs,
                              uint64_t width, int reenc_head, uint64_t ah1r, uint64_t ah1invr, int side,
                              uint64_t aoid, ahead_bat* out, uint64_t cap, ahead_errvec* errs) {
    if (!ctx || !l || !r || !out) return AHEAD_BAD_ARG;
    if (r->count && (!r_strs || width == 0))
        return fail(ctx, AHEAD_BAD_ARG, "hashjoinAN(str): right string slots required");
    // The join itself, with the right tail as the void row ids 0..n-1: its
    // tail output is the matched right row, in the reference's emit order.
    ahead_bat rr = *r;
    rr.tail = ahead_col{};
    rr.tail.type = AHEAD_VOID;
    uint32_t* rows = nullptr;
    const uint64_t rcap = (out->head.data && out->tail.data) ? cap : 0;
    if (rcap) AHEAD_CUDA(ctx, cudaMallocAsync((void**)&rows, rcap * 4, ctx->stream));
    ahead_bat o = *out;
    o.tail.data = rows;
    int rc = ahead_gpu_hashjoin_an(ctx, l, &rr, reenc_head, ah1r, ah1invr, 0, 1, 1, side, aoid, &o, rcap, errs);
    if (rc == AHEAD_OK && o.count) {
        // right side hashed: the reference decodes the left head before it
        // emits it (hashjoinAN.tcc:339,352)
        const bool decode = side == AHEAD_HASH_RIGHT && type_encoded(l->head.type);
        const uint64_t ainv = decode ? l->head.Ainv : 1;
        const int hw = type_width(o.head.type);
        const uint64_t n = o.count;
        const uint64_t want = (n + 255) / 256;
        const unsigned grid = (unsigned)(want < (uint64_t)ctx->num_sms * 8 ? want : (uint64_t)ctx->num_sms * 8);
        str_gather_kernel<<<grid, 256, 0, ctx->stream>>>(rows, n, r_strs, width, (char*)out->tail.data, decode,
                                                         ainv, out->head.data, hw);
        ctx->launches += 1;
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "hashjoinAN(str) gather");
    }
    if (rc == AHEAD_OK && side == AHEAD_HASH_LEFT && l->tail.type == AHEAD_RESTINY && errs && l->count && r->count) {
        // The string join's left build checks the restiny code without a cast
        // (hashjoinAN.tcc:290): the u16 product is promoted to int, not reduced
        // mod 2^16, and the compiled reference wraps it to 32 bits.
        rc = restiny_promoted_check(ctx, (const uint16_t*)l->tail.data, l->count,
                                    (uint32_t)(l->tail.Ainv & 0xFFFF), (uint32_t)(l->tail.unenc_max & 0xFFFF), aoid,
                                    &errs[1]);
    }
    if (rows) cudaFreeAsync(rows, ctx->stream);
    out->head = o.head;
    out->head.data = o.head.data;
    out->count = o.count;
    const void* tdata = out->tail.data;
    set_meta(&out->tail, AHEAD_STR, 0, 0, 0, 0);
    out->tail.data = const_cast<void*>(tdata);
    if (errs) {
        errs[3].present = 0;
        errs[3].count = 0;
    }
    return rc;
}

int ahead_gpu_hashjoin_an(ahead_ctx* ctx, const ahead_bat* l, const ahead_bat* r, int reenc_head, uint64_t ah1r,
                          uint64_t ah1invr, int reenc_tail, uint64_t at2r, uint64_t at2invr, int side, uint64_t aoid,
                          ahead_bat* out, uint64_t cap, ahead_errvec* errs) {
    if (!ctx || !l || !r || !out) return AHEAD_BAD_ARG;
    const int H1 = l->head.type, T1 = l->tail.type, H2 = r->head.type, T2 = r->tail.type;
    if (!(H1 == AHEAD_VOID || H1 == AHEAD_RESOID) || !(T2 == AHEAD_VOID || T2 == AHEAD_RESOID) || !small_res(T1) ||
        !small_res(H2))
        return fail(ctx, AHEAD_BAD_ARG, "hashjoinAN: (void|resoid, restiny|resshort|resint) x (res*, void|resoid)");
    if (reenc_tail && !reenc_head) return fail(ctx, AHEAD_BAD_ARG, "hashjoinAN: tail re-encoding needs head re-encoding");
    const int eH1 = type_encoded(H1), eT2 = type_encoded(T2);
    const int wh1e = type_width(type_encoded_of(H1)), wt2e = type_width(type_encoded_of(T2));
    const uint64_t AH1Inv = eH1 ? l->head.Ainv & wmask(wh1e) : 0, AT2Inv = eT2 ? r->tail.Ainv & wmask(wt2e) : 0;
    const uint64_t fH1 = eH1 ? mulw(ah1r, AH1Inv, type_width(H1)) : (ah1r & 0xffffffffull);
    const uint64_t fT2 = eT2 ? mulw(at2r, AT2Inv, type_width(T2)) : (at2r & 0xffffffffull);
    const int oH = reenc_head ? type_encoded_of(H1) : type_select_of(H1);
    const int oT = reenc_tail ? type_encoded_of(T2) : type_select_of(T2);
    if (reenc_head) {
        set_meta(&out->head, oH, ah1r, ah1invr, l->head.unenc_max, 0);
        if (reenc_tail) set_meta(&out->tail, oT, at2r, at2invr, r->tail.unenc_max, 0);
        else set_meta(&out->tail, oT, r->tail.A, r->tail.Ainv, r->tail.unenc_max, 0);
    } else {
        copy_meta(&out->head, oH, &l->head);
        copy_meta(&out->tail, oT, &r->tail);
    }
    set_errs_present(errs, eH1, 1, 1, eT2);
    out->count = 0;
    OpScope s(ctx);
    const uint64_t nl = l->count, nr = r->count;
    const bool both = nl > 0 && nr > 0;
    if (!both) return s.empty(out, cap, true);
    const bool left = side == AHEAD_HASH_LEFT;
    const uint64_t nb = left ? nl : nr, np = left ? nr : nl;
    const int bt1 = type_base_width(T1), bh2 = type_base_width(H2);
    const int larger = bt1 > bh2 ? bt1 : bh2;
    JoinOut o;
    o.fh = fH1;
    o.ft = fT2;
    o.cap = (out->head.data && out->tail.data) ? cap : 0;
    o.oh = out->head.data;
    o.ot = out->tail.data;
    o.rh = reenc_head;
    o.rt = reenc_tail;
    o.ohw = type_width(oH);
    o.otw = type_width(oT);
    o.probe_is_head = !left;
    o.pcol = dcol(left ? r->tail : l->head);
    o.bcol = dcol(left ? l->head : r->tail);
    const KeyCfg bk = left ? key_cfg(l->tail, 1, bt1, bt1, false) : key_cfg(r->head, 1, bh2, bh2, false);
    const KeyCfg pk = left ? key_cfg(r->head, 1, bt1, larger, true) : key_cfg(l->tail, 1, bh2, larger, true);
    // the column check of error vector k (head1, tail1, head2, tail2) into counter 1 + k
    auto check = [&](int k) {
        if (k == 0 && eH1)
            run_colcheck(s, l->head, nl, AH1Inv, l->head.unenc_max & wmask(wh1e), wh1e, aoid, ev(errs, 0), 1);
        if (k == 1)
            run_colcheck(s, l->tail, nl, l->tail.Ainv & wmask(type_width(T1)),
                         l->tail.unenc_max & wmask(type_width(T1)), type_width(T1), aoid, ev(errs, 1), 2);
        if (k == 2)
            run_colcheck(s, r->head, nr, r->head.Ainv & wmask(type_width(H2)),
                         r->head.unenc_max & wmask(type_width(H2)), type_width(H2), aoid, ev(errs, 2), 3);
        if (k == 3 && eT2)
            run_colcheck(s, r->tail, nr, AT2Inv, r->tail.unenc_max & wmask(wt2e), wt2e, aoid, ev(errs, 3), 4);
    };
    // error vectors of the probe's key and output column, and the build's
    const int vpk = left ? 2 : 1, vpo = left ? 3 : 0, vbk = left ? 1 : 2, vbo = left ? 0 : 3;
    ErrList kerr, verr;
    int rc = AHEAD_OK;
    bool direct = dj_possible(nb, np);
    if (direct) {
        rc = s.reserve(dj_scratch(nb, np));
        if (rc && rc != AHEAD_NO_MEMORY) return rc;
        direct = !rc;  // (device memory short: the table may need less)
    }
    if (direct) {
        rc = run_direct_join<true>(s, bk, nb, pk, np, o, aoid, ev(errs, vpk), ev(errs, vpo), &kerr, &verr,
                                   s.sized(out, cap) ? out : nullptr);
        if (rc) return rc;
    }
    if (direct && !s.counter(kDjBad)) {
        out->count = s.counter(0);
        if (errs) {
            errs[vpk].count = s.counter(1);
            if (errs[vpo].present) errs[vpo].count = s.counter(2);
            const bool okk = settle_err_list(s, kerr, kDjBuildKey, aoid, ev(errs, vbk));
            const bool okv = !errs[vbo].present || settle_err_list(s, verr, kDjBuildVal, aoid, ev(errs, vbo));
            if (!okk || !okv) {  // a build column with many corrupt codes
                rc = s.reserve(2 * colcheck_scratch(nb));
                if (rc) return rc;
                if (!okk) check(vbk);
                if (!okv) check(vbo);
                rc = s.finish(5);
                if (rc) return rc;
                if (!okk) errs[vbk].count = s.counter(1 + vbk);
                if (!okv) errs[vbo].count = s.counter(1 + vbo);
            }
        }
        rc = s.wait();
        if (rc) return rc;
        return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
    }
    rc = s.reserve(join_scratch(nb, np) + colcheck_scratch(nl) * 2 + colcheck_scratch(nr) * 2);
    if (rc) return rc;
    const bool sized = s.sized(out, cap);
    // (build columns that the bitmap form has just found clean are not read again)
    const bool clean_key = direct && !s.counter(kDjBuildKey), clean_val = direct && !s.counter(kDjBuildVal);
    rc = run_hash_join(s, bk, nb, pk, np, o, sized ? out : nullptr);
    if (rc) return rc;
    for (int k = 0; k < 4; ++k)
        if (!(clean_key && k == vbk) && !(clean_val && k == vbo)) check(k);
    rc = s.finish(5);
    if (rc) return rc;
    if (!sized) out->count = s.counter(0);
    if (errs)
        for (int k = 0; k < 4; ++k)
            if (errs[k].present) errs[k].count = s.counter(1 + k);
    return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_hashjoin(ahead_ctx* ctx, const ahead_bat* l, const ahead_bat* r, int side, ahead_bat* out,
                       uint64_t cap) {
    if (!ctx || !l || !r || !out) return AHEAD_BAD_ARG;
    const int H1 = l->head.type, T1 = l->tail.type, H2 = r->head.type, T2 = r->tail.type;
    if (!(H1 == AHEAD_VOID || H1 == AHEAD_OID) || !(T2 == AHEAD_VOID || T2 == AHEAD_OID) || T1 != H2 ||
        T1 == AHEAD_VOID || T1 == AHEAD_OID || T1 == AHEAD_BIGINT || T1 == AHEAD_RESBIGINT || T1 == AHEAD_RESOID)
        return fail(ctx, AHEAD_BAD_ARG, "hashjoin: (void|oid, K) x (K, void|oid) with a 1/2/4-byte or res key K");
    copy_meta(&out->head, type_select_of(H1), &l->head);
    copy_meta(&out->tail, type_select_of(T2), &r->tail);
    out->count = 0;
    OpScope s(ctx);
    const uint64_t nl = l->count, nr = r->count;
    const bool both = nl > 0 && nr > 0;
    const uint64_t nb = side == AHEAD_HASH_LEFT ? nl : nr, np = side == AHEAD_HASH_LEFT ? nr : nl;
    if (!both) return s.empty(out, cap, true);
    const int w = type_width(T1);
    JoinOut o;
    o.fh = o.ft = 1;
    o.cap = (out->head.data && out->tail.data) ? cap : 0;
    o.oh = out->head.data;
    o.ot = out->tail.data;
    o.rh = o.rt = 0;
    o.ohw = type_width(type_select_of(H1));
    o.otw = type_width(type_select_of(T2));
    const KeyCfg bk = key_cfg(side == AHEAD_HASH_LEFT ? l->tail : r->head, 0, w, w, false);
    const KeyCfg pk = key_cfg(side == AHEAD_HASH_LEFT ? r->head : l->tail, 0, w, w, false);
    o.probe_is_head = side != AHEAD_HASH_LEFT;
    o.pcol = dcol(side == AHEAD_HASH_LEFT ? r->tail : l->head);
    o.bcol = dcol(side == AHEAD_HASH_LEFT ? l->head : r->tail);
    int rc = AHEAD_OK;
    bool direct = w < 8 && dj_possible(nb, np);  // (8-byte keys are raw codes)
    if (direct) {
        rc = s.reserve(dj_scratch(nb, np));
        if (rc && rc != AHEAD_NO_MEMORY) return rc;
        direct = !rc;
    }
    if (direct) {
        ErrList kerr, verr;
        rc = run_direct_join<false>(s, bk, nb, pk, np, o, 0, nullptr, nullptr, &kerr, &verr,
                                    s.sized(out, cap) ? out : nullptr);
        if (rc) return rc;
        if (!s.counter(kDjBad)) {
            out->count = s.counter(0);
            return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
        }
    }
    rc = s.reserve(join_scratch(nb, np));
    if (rc) return rc;
    const bool sized = s.sized(out, cap);
    rc = run_hash_join(s, bk, nb, pk, np, o, sized ? out : nullptr);
    if (rc) return rc;
    if (sized) return s.wait();
    rc = s.finish(1);
    if (rc) return rc;
    out->count = s.counter(0);
    return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_matchjoin_an(ahead_ctx* ctx, const ahead_bat* a, const ahead_bat* b, int reenc, uint64_t ah1r,
                           uint64_t ah1invr, uint64_t at2r, uint64_t at2invr, uint64_t aoid, ahead_bat* out,
                           uint64_t cap, ahead_errvec* errs) {
    if (!ctx || !a || !b || !out) return AHEAD_BAD_ARG;
    const int H1 = a->head.type, T1 = a->tail.type, H2 = b->head.type, T2 = b->tail.type;
    const bool vv = T1 == AHEAD_VOID && H2 == AHEAD_VOID, rv = T1 == AHEAD_RESOID && H2 == AHEAD_VOID;
    const bool gm = T1 == AHEAD_RESOID && H2 == AHEAD_RESOID, mv = T1 == AHEAD_VOID && H2 == AHEAD_RESOID;
    if (!(H1 == AHEAD_VOID || H1 == AHEAD_RESOID || H1 == AHEAD_RESINT) || !(vv || rv || gm || mv) ||
        (H1 == AHEAD_VOID && T1 == AHEAD_VOID) || (T2 == AHEAD_VOID && !gm) ||
        !(T2 == AHEAD_VOID || type_encoded(T2)))
        return fail(ctx, AHEAD_BAD_ARG, "matchjoinAN: unsupported type combination");
    if (reenc && (H1 == AHEAD_VOID || T2 == AHEAD_VOID))
        return fail(ctx, AHEAD_UNSUPPORTED, "matchjoinAN: re-encoding with a void head or tail");
    DCol h1 = dcol(a->head), t1 = dcol(a->tail), h2 = dcol(b->head), t2 = dcol(b->tail);
    const uint64_t fH1 = dec_if_host(h1, ah1r), fT2 = dec_if_host(t2, at2r);
    const int oH = reenc ? type_encoded_of(H1) : type_select_of(H1);
    const int oT = reenc ? type_encoded_of(T2) : type_select_of(T2);
    if (reenc) {
        set_meta(&out->head, oH, ah1r, ah1invr, a->head.unenc_max, 0);
        set_meta(&out->tail, oT, at2r, at2invr, b->tail.unenc_max, 0);
    } else {
        copy_meta(&out->head, oH, &a->head);
        copy_meta(&out->tail, oT, &b->tail);
    }
    out->count = 0;
    const uint64_t n1 = a->count, n2 = b->count;
    const uint64_t ocap = (out->head.data && out->tail.data) ? cap : 0;
    OpScope s(ctx);
    if (rv) {
        set_errs_present(errs, type_encoded(H1), 1, 0, type_encoded(T2));
        const uint64_t sz = (uint32_t)b->count;  // BAT::size() is an oid_t
        int rc;
        if (pos_one_pass(n1, ocap, sz)) {
            PosArgs pa{};
            pa.base = (const char*)a->tail.data;
            pa.n = n1;
            pa.inv = a->tail.Ainv;
            pa.sz = sz;
            pa.h1c = h1;
            pa.t2c = t2;
            pa.fh = fH1;
            pa.ft = fT2;
            pa.oh = out->head.data;
            pa.ot = out->tail.data;
            pa.ohw = type_width(oH);
            pa.otw = type_width(oT);
            pa.reenc = reenc;
            pa.head_err = type_encoded(H1);
            pa.t2enc = type_encoded(T2);
            pa.w2 = t2.width;
            uint64_t kept = 0;
            rc = run_pos_join<true, false>(s, pa, &a->head, aoid, h1.umax == 0, ev(errs, 0), ev(errs, 1), ev(errs, 3),
                                           &kept);
            if (rc != AHEAD_UNSUPPORTED) {
                if (rc == AHEAD_OK) out->count = kept;
                return rc;
            }
        }
        rc = s.reserve(compact_scratch<MjPosOp<true>>(n1));
        if (rc) return rc;
        MjPosOp<true> op;
        op.base = (const char*)a->tail.data;
        op.h1c = h1;
        op.t2c = t2;
        op.at1inv = a->tail.Ainv;
        op.ah1inv = type_encoded(H1) ? a->head.Ainv : 0;
        op.ah1max = a->head.unenc_max;
        op.sz = sz;
        op.fh = fH1;
        op.ft = fT2;
        op.cap = ocap;
        op.aoid = aoid;
        op.e1 = edata(ev(errs, 0));
        op.e2 = edata(ev(errs, 1));
        op.e4 = edata(ev(errs, 3));
        op.ec1 = ecap(ev(errs, 0));
        op.ec2 = ecap(ev(errs, 1));
        op.ec4 = ecap(ev(errs, 3));
        op.acc = nullptr;
        op.oh = out->head.data;
        op.ot = out->tail.data;
        op.ohw = type_width(oH);
        op.otw = type_width(oT);
        op.reenc = reenc;
        op.h1enc = type_encoded(H1);
        op.t2enc = type_encoded(T2);
        run_compact(s, op, n1, 0);
        rc = s.finish(4);
        if (rc) return rc;
        out->count = s.counter(0);
        if (errs) {
            if (errs[0].present) errs[0].count = s.counter(1);
            errs[1].count = s.counter(2);
            if (errs[3].present) errs[3].count = s.counter(3);
        }
        return out->count > cap || s.sized(out, cap) ? AHEAD_CAPACITY : AHEAD_OK;
    }
    if (vv) {
        set_errs_present(errs, type_encoded(H1), 0, 0, type_encoded(T2));
        uint64_t p1 = 0, p2 = 0, m = 0;
        if (n1 && n2) {
            if (a->tail.seqbase < b->head.seqbase) p1 = vv_skip(a->tail.seqbase, b->head.seqbase, n1);
            else if (a->tail.seqbase > b->head.seqbase) p2 = vv_skip(b->head.seqbase, a->tail.seqbase, n2);
            m = (n1 - p1) < (n2 - p2) ? (n1 - p1) : (n2 - p2);
        }
        int rc = s.reserve(colcheck_scratch(p1 + m) + colcheck_scratch(p2 + m));
        if (rc) return rc;
        if (m && ocap)
            zip_kernel<<<grid_for(m, 256), 256, 0, ctx->stream>>>(h1, t2, p1, p2, m, reenc, fH1, fT2, out->head.data,
                                                                   type_width(oH), out->tail.data, type_width(oT),
                                                                   ocap);
        if (n1 && n2) {
            if (type_encoded(H1))
                run_colcheck(s, a->head, p1 + m, h1.ainv, h1.umax, type_width(H1), aoid, ev(errs, 0), 0);
            if (type_encoded(T2))
                run_colcheck(s, b->tail, p2 + m, t2.ainv, t2.umax, type_width(T2), aoid, ev(errs, 3), 1);
        }
        rc = s.finish(2);
        if (rc) return rc;
        out->count = m;
        if (errs) {
            if (errs[0].present) errs[0].count = (n1 && n2) ? s.counter(0) : 0;
            if (errs[3].present) errs[3].count = (n1 && n2) ? s.counter(1) : 0;
        }
        return m > cap || s.sized(out, cap) ? AHEAD_CAPACITY : AHEAD_OK;
    }
    // general merge (gm) or (void tail, resoid head) merge (mv)
    set_errs_present(errs, type_encoded(H1), type_encoded(T1), type_encoded(H2), type_encoded(T2));
    if (!n1 || !n2) return s.empty(out, cap, true);
    int rc;
    const int dw = type_width(T1 == AHEAD_VOID ? H1 : T1);  // 8: the head of a void list is encoded
    {
        const uint64_t nt1 = (n1 + kMeTile - 1) / kMeTile, nt2 = (n2 + kMeTile - 1) / kMeTile;
        rc = s.reserve(merge_scratch(n1) + (nt1 + nt2) * 24 + 4096);
        if (rc) return rc;
        rc = run_merge(s, t1, h1, h2, t2, n1, n2, true, dw, reenc, fH1, fT2, out, cap);
        if (rc) return rc;
        const uint32_t flag = (uint32_t)s.counter(kMergeFlag);
        if (!(flag & 1u)) {
            out->count = s.counter(0);
            if (flag & 2u) {
                // corrupt values in ordered inputs: the loop's error positions, per row
                MergeErrs me;
                me.h1 = h1;
                me.t1 = t1;
                me.h2 = h2;
                me.t2 = t2;
                me.n1 = n1;
                me.n2 = n2;
                me.aoid = aoid;
                me.eh1 = type_encoded(H1);
                me.et1 = type_encoded(T1);
                me.eh2 = type_encoded(H2);
                me.et2 = type_encoded(T2);
                uint64_t* l1m = (uint64_t*)s.alloc(8);
                me.l1m = l1m;
                merge_last_kernel<<<1, 1, 0, ctx->stream>>>(me, l1m);
                s.launched();
                for (int side = 0; side < 2; ++side) {
                    const uint64_t n = side ? n2 : n1;
                    const uint64_t nt = side ? nt2 : nt1;
                    auto* tcount = (uint32_t*)s.alloc(nt * 8);
                    auto* toff = (uint64_t*)s.alloc(nt * 16);
                    merge_err_count_kernel<<<(uint32_t)nt, kMeThreads, 0, ctx->stream>>>(me, side, n, tcount);
                    merge_err_scan_kernel<<<1, kMeThreads, 0, ctx->stream>>>(tcount, toff, (uint32_t)nt,
                                                                             s.d_counters + 1 + 2 * side);
                    const ahead_errvec* va = ev(errs, 2 * side);
                    const ahead_errvec* vb = ev(errs, 2 * side + 1);
                    merge_err_write_kernel<<<(uint32_t)nt, kMeThreads, 0, ctx->stream>>>(
                        me, side, n, toff, edata(va), ecap(va), edata(vb), ecap(vb));
                    s.launched(3);
                }
                rc = s.finish(5);
                if (rc) return rc;
                if (errs)
                    for (int k = 0; k < 4; ++k)
                        if (errs[k].present) errs[k].count = s.counter(1 + k);
            }
            return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
        }
    }
    rc = s.reserve(0);
    if (rc) return rc;
    rc = seq_columns(s, out, n1, n2, cap);
    if (rc) return rc;
    MergeSeq m;
    m.h1 = h1;
    m.t1 = t1;
    m.h2 = h2;
    m.t2 = t2;
    m.n1 = n1;
    m.n2 = n2;
    m.fh = fH1;
    m.ft = fT2;
    m.aoid = aoid;
    m.cap = (out->head.data && out->tail.data) ? cap : 0;
    for (int k = 0; k < 4; ++k) {
        m.e[k] = edata(ev(errs, k));
        m.ecap[k] = ecap(ev(errs, k));
    }
    m.oh = out->head.data;
    m.ot = out->tail.data;
    m.ohw = type_width(oH);
    m.otw = type_width(oT);
    m.reenc = reenc;
    m.checked = 1;
    merge_seq_kernel<<<1, 32, 0, ctx->stream>>>(m, s.d_counters);
    s.launched();
    rc = s.finish(5);
    if (rc) return rc;
    out->count = s.counter(0);
    if (errs)
        for (int k = 0; k < 4; ++k)
            if (errs[k].present) errs[k].count = s.counter(1 + k);
    return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_matchjoin(ahead_ctx* ctx, const ahead_bat* a, const ahead_bat* b, ahead_bat* out, uint64_t cap) {
    if (!ctx || !a || !b || !out) return AHEAD_BAD_ARG;
    const int H1 = a->head.type, T1 = a->tail.type, H2 = b->head.type, T2 = b->tail.type;
    auto oidish = [](int t) { return t == AHEAD_VOID || t == AHEAD_OID; };
    // heads instantiated in Normal/matchjoin.hpp:36-50 (strings aside)
    if (H1 == AHEAD_RESOID || !oidish(T1) || !oidish(H2) || T2 == AHEAD_VOID || T2 == AHEAD_RESOID ||
        (H1 == AHEAD_VOID && T1 == AHEAD_VOID))
        return fail(ctx, AHEAD_BAD_ARG, "matchjoin: unsupported type combination");
    copy_meta(&out->head, type_select_of(H1), &a->head);
    copy_meta(&out->tail, type_select_of(T2), &b->tail);
    out->count = 0;
    const uint64_t n1 = a->count, n2 = b->count;
    const uint64_t ocap = (out->head.data && out->tail.data) ? cap : 0;
    DCol h1 = dcol(a->head), t1 = dcol(a->tail), h2 = dcol(b->head), t2 = dcol(b->tail);
    OpScope s(ctx);
    if (T1 == AHEAD_VOID && H2 == AHEAD_VOID) {
        uint64_t p1 = 0, p2 = 0, m = 0;
        if (n1 && n2) {
            if (a->tail.seqbase < b->head.seqbase) p1 = vv_skip(a->tail.seqbase, b->head.seqbase, n1);
            else if (a->tail.seqbase > b->head.seqbase) p2 = vv_skip(b->head.seqbase, a->tail.seqbase, n2);
            m = (n1 - p1) < (n2 - p2) ? (n1 - p1) : (n2 - p2);
        }
        int rc = s.reserve(0);
        if (rc) return rc;
        if (m && ocap) {
            zip_kernel<<<grid_for(m, 256), 256, 0, ctx->stream>>>(h1, t2, p1, p2, m, 0, 1, 1, out->head.data,
                                                                   type_width(type_select_of(H1)), out->tail.data,
                                                                   type_width(type_select_of(T2)), ocap);
            s.launched();
        }
        rc = s.finish(0);
        if (rc) return rc;
        out->count = m;
        return m > cap || s.sized(out, cap) ? AHEAD_CAPACITY : AHEAD_OK;
    }
    if (T1 == AHEAD_OID && H2 == AHEAD_VOID) {
        int rc;
        if (pos_one_pass(n1, ocap, n2)) {
            PosArgs pa{};
            pa.base = (const char*)a->tail.data;
            pa.n = n1;
            pa.sz = n2;
            pa.h1c = h1;
            pa.t2c = t2;
            pa.oh = out->head.data;
            pa.ot = out->tail.data;
            pa.ohw = type_width(type_select_of(H1));
            pa.otw = type_width(type_select_of(T2));
            uint64_t kept = 0;
            rc = run_pos_join<false, false>(s, pa, nullptr, 0, false, nullptr, nullptr, nullptr, &kept);
            if (rc != AHEAD_UNSUPPORTED) {
                if (rc == AHEAD_OK) out->count = kept;
                return rc;
            }
        }
        rc = s.reserve(compact_scratch<MjPosOp<false>>(n1));
        if (rc) return rc;
        MjPosOp<false> op{};
        op.base = (const char*)a->tail.data;
        op.h1c = h1;
        op.t2c = t2;
        op.sz = n2;
        op.cap = ocap;
        op.acc = nullptr;
        op.oh = out->head.data;
        op.ot = out->tail.data;
        op.ohw = type_width(type_select_of(H1));
        op.otw = type_width(type_select_of(T2));
        run_compact(s, op, n1, 0);
        rc = s.finish(1);
        if (rc) return rc;
        out->count = n1 ? s.counter(0) : 0;
        return out->count > cap || s.sized(out, cap) ? AHEAD_CAPACITY : AHEAD_OK;
    }
    // merge on plain oid values: strictly increasing keys intersect in parallel
    // (driving column of 2, 4 or 8 bytes); anything else replays the loop
    const int dw = type_width(T1 == AHEAD_VOID ? H1 : T1);
    if (!n1 || !n2) return s.empty(out, cap, true);
    if (dw >= 2) {
        int rc = s.reserve(merge_scratch(n1));
        if (rc) return rc;
        DCol k1 = t1, k2 = h2, v1 = h1, v2 = t2;
        k1.enc = k2.enc = v1.enc = v2.enc = 0;  // plain values
        rc = run_merge(s, k1, v1, k2, v2, n1, n2, false, dw, 0, 1, 1, out, cap);
        if (rc) return rc;
        if (!(s.counter(kMergeFlag) & 1u)) {
            out->count = s.counter(0);
            return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
        }
    }
    int rc = s.reserve(0);
    if (rc) return rc;
    rc = seq_columns(s, out, n1, n2, cap);
    if (rc) return rc;
    MergeSeq m{};
    m.h1 = h1;
    m.t1 = t1;
    m.h2 = h2;
    m.t2 = t2;
    m.n1 = n1;
    m.n2 = n2;
    m.cap = (out->head.data && out->tail.data) ? cap : 0;
    m.oh = out->head.data;
    m.ot = out->tail.data;
    m.ohw = type_width(type_select_of(H1));
    m.otw = type_width(type_select_of(T2));
    m.checked = 0;
    merge_seq_kernel<<<1, 32, 0, ctx->stream>>>(m, s.d_counters);
    s.launched();
    rc = s.finish(1);
    if (rc) return rc;
    out->count = s.counter(0);
    return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_fetchjoin_an(ahead_ctx* ctx, const ahead_bat* a, const ahead_bat* b, int reenc, uint64_t atr,
                           uint64_t atrinv, uint64_t aoid, ahead_bat* out, uint64_t cap, ahead_errvec* errs) {
    if (!ctx || !a || !b || !out) return AHEAD_BAD_ARG;
    const int T2 = b->tail.type;
    if (a->head.type != AHEAD_VOID || a->tail.type != AHEAD_RESOID || b->head.type != AHEAD_VOID || !type_encoded(T2))
        return fail(ctx, AHEAD_BAD_ARG, "fetchjoinAN: (void, resoid) x (void, AN tail) required");
    const int w = type_width(T2);
    copy_meta(&out->head, AHEAD_VOID, &a->head);
    copy_meta(&out->tail, T2, &b->tail);
    uint64_t fac = 1;
    if (reenc) {
        out->tail.A = (uint16_t)atr;
        out->tail.Ainv = atrinv;
        fac = mulw(atr, inv_pow2(b->tail.A, 8 * w), w);
    }
    if (errs) {
        ev_begin(&errs[0], 1);
        ev_begin(&errs[1], 1);
    }
    out->count = 0;
    OpScope s(ctx);
    int rc;
    if (pos_one_pass(a->count, out->tail.data ? cap : 0, b->count)) {
        PosArgs pa{};
        pa.base = (const char*)a->tail.data;
        pa.n = a->count;
        pa.inv = a->tail.Ainv;
        pa.sz = b->count;
        pa.t2c = dcol(b->tail);
        pa.ft = fac;
        pa.ot = out->tail.data;
        pa.otw = w;
        pa.reenc = reenc;
        pa.t2enc = 1;
        pa.w2 = w;
        uint64_t kept = 0;
        rc = run_pos_join<true, true>(s, pa, nullptr, aoid, false, nullptr, ev(errs, 0), ev(errs, 1), &kept);
        if (rc != AHEAD_UNSUPPORTED) {
            if (rc == AHEAD_OK) out->count = kept;
            return rc;
        }
    }
    rc = s.reserve(compact_scratch<FetchOp<true>>(a->count));
    if (rc) return rc;
    FetchOp<true> op;
    op.base = (const char*)a->tail.data;
    op.t2c = dcol(b->tail);
    op.at1inv = a->tail.Ainv;
    op.at2inv = b->tail.Ainv & wmask(w);
    op.at2max = b->tail.unenc_max & wmask(w);
    op.vsz = b->count;
    op.fac = fac;
    op.cap = out->tail.data ? cap : 0;
    op.aoid = aoid;
    op.e1 = edata(ev(errs, 0));
    op.e2 = edata(ev(errs, 1));
    op.ec1 = ecap(ev(errs, 0));
    op.ec2 = ecap(ev(errs, 1));
    op.acc = nullptr;
    op.ot = out->tail.data;
    op.otw = w;
    op.reenc = reenc;
    op.w2 = w;
    run_compact(s, op, a->count, 0);
    rc = s.finish(3);
    if (rc) return rc;
    out->count = a->count ? s.counter(0) : 0;
    if (errs) {
        errs[0].count = a->count ? s.counter(1) : 0;
        errs[1].count = a->count ? s.counter(2) : 0;
    }
    return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_fetchjoin(ahead_ctx* ctx, const ahead_bat* a, const ahead_bat* b, ahead_bat* out, uint64_t cap) {
    if (!ctx || !a || !b || !out) return AHEAD_BAD_ARG;
    const int T2 = b->tail.type;
    if (a->head.type != AHEAD_VOID || a->tail.type != AHEAD_OID || b->head.type != AHEAD_VOID || T2 == AHEAD_VOID ||
        T2 == AHEAD_RESOID)
        return fail(ctx, AHEAD_BAD_ARG, "fetchjoin: (void, oid) x (void, value) required");
    copy_meta(&out->head, AHEAD_VOID, &a->head);
    copy_meta(&out->tail, T2, &b->tail);
    out->count = 0;
    OpScope s(ctx);
    int rc;
    if (pos_one_pass(a->count, out->tail.data ? cap : 0, b->count)) {
        PosArgs pa{};
        pa.base = (const char*)a->tail.data;
        pa.n = a->count;
        pa.sz = b->count;
        pa.t2c = dcol(b->tail);
        pa.ot = out->tail.data;
        pa.otw = type_width(T2);
        uint64_t kept = 0;
        rc = run_pos_join<false, true>(s, pa, nullptr, 0, false, nullptr, nullptr, nullptr, &kept);
        if (rc != AHEAD_UNSUPPORTED) {
            if (rc == AHEAD_OK) out->count = kept;
            return rc;
        }
    }
    rc = s.reserve(compact_scratch<FetchOp<false>>(a->count));
    if (rc) return rc;
    FetchOp<false> op{};
    op.base = (const char*)a->tail.data;
    op.t2c = dcol(b->tail);
    op.vsz = b->count;
    op.fac = 1;
    op.cap = out->tail.data ? cap : 0;
    op.acc = nullptr;
    op.ot = out->tail.data;
    op.otw = type_width(T2);
    op.w2 = type_width(T2);
    run_compact(s, op, a->count, 0);
    rc = s.finish(1);
    if (rc) return rc;
    out->count = a->count ? s.counter(0) : 0;
    return out->count > cap ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_fetchjoin_str_an(ahead_ctx* ctx, const ahead_bat* a, const char* strs, uint64_t width, uint64_t count,
                               uint64_t aoid, char* out, uint64_t cap, uint64_t* n_out, ahead_errvec* errs) {
    if (!ctx || !a || !n_out || !width) return AHEAD_BAD_ARG;
    if (a->head.type != AHEAD_VOID || a->tail.type != AHEAD_RESOID || (count && !strs) || count >= (1ull << 32))
        return fail(ctx, AHEAD_BAD_ARG, "fetchjoinAN(str): (void, resoid) OIDs and string slots required");
    if (errs) {
        ev_begin(&errs[0], 1);
        ev_begin(&errs[1], 0);
    }
    *n_out = 0;
    const uint64_t n = a->count;
    OpScope s(ctx);
    int rc = s.reserve(compact_scratch<FetchStrOp>(n) + n * 4 + 4096);
    if (rc) return rc;
    uint32_t* rows = (uint32_t*)s.alloc((n ? n : 1) * 4);
    FetchStrOp op;
    op.base = (const char*)a->tail.data;
    op.ainv = a->tail.Ainv;
    op.count = count;
    op.aoid = aoid;
    op.cap = n;
    op.rows = rows;
    op.err = edata(errs);
    op.errcap = ecap(errs);
    op.acc = nullptr;
    run_compact(s, op, n, 0);
    rc = s.finish(2);
    if (rc) return rc;
    const uint64_t kept = s.counter(0);
    *n_out = kept;
    if (errs) errs[0].count = s.counter(1);
    if (kept > cap) return AHEAD_CAPACITY;
    return gather_str_rows(ctx, rows, kept, strs, width, out);
}

int ahead_gpu_fetchjoin_str(ahead_ctx* ctx, const ahead_bat* a, const char* strs, uint64_t width, uint64_t count,
                            char* out, uint64_t cap, uint64_t* n_out) {
    if (!ctx || !a || !n_out || !width) return AHEAD_BAD_ARG;
    if (a->head.type != AHEAD_VOID || a->tail.type != AHEAD_OID || (count && !strs))
        return fail(ctx, AHEAD_BAD_ARG, "fetchjoin(str): (void, oid) OIDs and string slots required");
    *n_out = 0;
    const uint64_t n = a->count;
    OpScope s(ctx);
    int rc = s.reserve(compact_scratch<FetchStrPlainOp>(n) + n * 4 + 4096);
    if (rc) return rc;
    uint32_t* rows = (uint32_t*)s.alloc((n ? n : 1) * 4);
    FetchStrPlainOp op;
    op.base = (const char*)a->tail.data;
    op.count = count;
    op.cap = n;
    op.rows = rows;
    op.acc = nullptr;
    run_compact(s, op, n, 0);
    rc = s.finish(1);
    if (rc) return rc;
    const uint64_t kept = s.counter(0);
    *n_out = kept;
    if (kept > cap) return AHEAD_CAPACITY;
    return gather_str_rows(ctx, rows, kept, strs, width, out);
}

}  // extern "C"
