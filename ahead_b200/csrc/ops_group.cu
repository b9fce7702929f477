// ops_group.cu -- groupbyAN (unary and binary), aggregate_sum_groupedAN, and
// their unencoded twins (groupby, aggregate_sum_grouped, aggregate_sum,
// arithmetic).
//
// Group ids are assigned in order of first occurrence, as the reference's
// dictionary loop does (lib/column_operators/AN/groupbyAN.tcc:70-91,
// 127-160).  On the GPU: every row lowers its key's first-row word (indexed by
// the key itself while the keys are small, else a slot of the hash table of
// hash.cuh); the groups are ranked by first row (a sort of the few, or a stable
// compaction of the rows that are their key's first row); a last pass writes
// every row's encoded group id.
#include "hash.cuh"
#include "ops_common.cuh"

using namespace ahead;

namespace {

struct GbKey {
    DCol tail, grp;
    uint64_t keymask, lmask, ngroups, gainv;
    int binary;
};

AHEAD_DEV uint64_t gb_key(const GbKey& k, uint64_t row) {
    const uint64_t t = dec_if(k.tail, load_at(k.tail, row), k.tail.ainv);
    if (!k.binary) return t & k.keymask;  // unary: the unencoded base type
    // binary: hash(t) * numGroups + g in the larger tail type (groupbyAN.tcc:144)
    const uint64_t g = load_at(k.grp, row) * k.gainv;
    return ((t & k.lmask) * (k.ngroups & k.lmask) + (g & k.lmask)) & k.lmask;
}

// A row's first look at the table takes the key word and the first row of the
// slot its key hashes to together (the slot is the key's own for nearly all
// rows), and a thread has U rows' looks in flight: at 12M rows of 70,000 dates the
// call took 555 us with a look at a time.  CHECK: the columns' AN checks
// ride along, corrupt rows go to short lists.
template <bool CHECK, int U>
__global__ void __launch_bounds__(256) gb_insert_kernel(HashTab h, GbKey k, uint64_t n, uint64_t gmax,
                                                        uint32_t* slot_of, uint32_t* first, ErrList terr,
                                                        ErrList gerr) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i0 < n; i0 += U * stride) {
        uint64_t key[U], seen[U];
        uint32_t slot[U], row[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + u * stride < n ? i0 + u * stride : i0;
            if (CHECK && i0 + u * stride < n) {
                if (dec_if(k.tail, load_at(k.tail, i), k.tail.ainv) > k.tail.umax) terr.add(i);
                if (k.binary && load_at(k.grp, i) * k.gainv > gmax) gerr.add(i);
            }
            key[u] = gb_key(k, i);
            slot[u] = ht_mix(key[u]) & h.mask;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            seen[u] = h.keys[slot[u]];
            row[u] = first[slot[u]];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + u * stride;
            if (i >= n) break;
            if (seen[u] != key[u] || key[u] == kEmptyKey) {
                slot[u] = ht_insert(h, key[u]);
                row[u] = first[slot[u]];
            }
            slot_of[i] = slot[u];
            if ((uint32_t)i < row[u]) atomicMin(&first[slot[u]], (uint32_t)i);  // (a stale word is only larger)
        }
    }
}

// Four rows a thread once every thread of the grid has them; fewer rows spread thinner.
template <bool CHECK>
void launch_gb_insert(const OpScope& s, const HashTab& h, const GbKey& k, uint64_t n, uint64_t gmax, uint32_t* slot_of,
                      uint32_t* first, const ErrList& terr, const ErrList& gerr) {
    const uint32_t grid = grid_for(n, 256);
    if (n >= (1u << 22))
        gb_insert_kernel<CHECK, 4><<<grid, 256, 0, s.ctx->stream>>>(h, k, n, gmax, slot_of, first, terr, gerr);
    else
        gb_insert_kernel<CHECK, 1><<<grid, 256, 0, s.ctx->stream>>>(h, k, n, gmax, slot_of, first, terr, gerr);
}

// Rows that are the first row of their group, in row order; the rank of such
// a row is its group id.  The driving column is the row's slot.
struct FirstOp {
    static constexpr int W = 4;
    static constexpr int NCH = 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = true;
    static constexpr bool EMIT_V = false;
    static constexpr int NOUT = 1;
    const char* base;
    const uint32_t* first;
    uint32_t* gid_of_slot;
    DCol head;
    uint64_t aoid, cap;
    uint64_t* firsts;
    uint64_t* acc;
    int decode_head;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t row, uint64_t&) const { return first[v] == (uint32_t)row ? 1u : 0u; }
    AHEAD_DEV uint64_t out0(int, uint64_t, uint64_t row) const { return row; }
    AHEAD_DEV uint64_t cap0() const { return ~0ull; }  // (every group gets its id)
    AHEAD_DEV void put0(int, uint64_t pos, uint64_t row) const {
        const uint32_t s = ((const uint32_t*)base)[row];
        gid_of_slot[s] = (uint32_t)pos;
        if (pos < cap) {
            const uint64_t h = load_at(head, row);
            // unary: raw head (groupbyAN.tcc:87); binary: decoded head (:153)
            firsts[pos] = (decode_head ? dec_if(head, h, head.ainv) : h) * aoid;
        }
    }
};

// Encoded group id of every row.  The binary group-by's dictionary stores the
// encoded id in an oid_t (groupbyAN.tcc:150): the first row of a group gets
// all 64 bits, later rows the low 32.
__global__ void gb_assign_kernel(const uint32_t* slot_of, const uint32_t* first, const uint32_t* gid_of_slot,
                                 uint64_t n, uint64_t aoid, int binary, uint64_t* gids, uint64_t cap) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n && i < cap;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = slot_of[i];
        const uint64_t v = (uint64_t)gid_of_slot[s] * aoid;
        gids[i] = (binary && first[s] != (uint32_t)i) ? (uint64_t)(uint32_t)v : v;
    }
}

// ---------------------------------------------------- small-key group-by
// Group keys are dictionary codes (years, categories, brands) or such a code
// times the number of groups so far plus a group id: small integers.  So the
// key indexes a table of first rows directly (`limit` 4-byte words: twice the
// rows, between 2^16 and 2^22, so clearing it costs no more than reading the
// inputs), without hashing, key words or probing, and neighbouring keys share
// L1 lines.  A row reads its key's word first and only lowers it when it would:
// once the seed block has seen the first rows, almost no row does an atomic.
// At 12M rows, year (7) then category (40): the hash table's one CAS and one
// atomicMin per row on a few words took 1,876 us for the two insert passes; the
// seed, insert, rank and assign kernels here take 61 us unary and 95 us binary
// (insert 22.8 and 46.2: 8 and 16 bytes a row at 4.2 TB/s, bound by HBM and
// the L1 gathers).  The columns' AN checks ride along: corrupt rows go to short
// lists.  A key at or above `limit` raises `over`, and the hash table takes the
// call: when a seed row has one, the grid's passes return at once.  What the
// attempt costs then (20-30 us: clearing the table, the seed, four empty launches,
// a wait) the table's insert pass gives back where it checks columns or many rows
// share a group.  12M rows, 40 wide keys 345 us (980 by the table alone before),
// 3M wide keys 1,200 (1,365), 70,000 dates 570 (557); unencoded 307 (909),
// 1,140 (1,285) and 525 (491); 1M rows, 250,000 wide keys: 147 (173), unencoded
// 138 (128).
constexpr uint32_t kGbMinLimit = 1u << 16, kGbMaxLimit = 1u << 22;
constexpr uint32_t kGbSort = 4096;  // groups ranked by one block's sort; more are ranked by the compaction
constexpr uint32_t kGbSeedRows = 4096;
constexpr uint32_t kNoRow = 0xffffffffu;

struct SmallGb {
    GbKey k;
    uint64_t n, gmax;        // gmax: largest valid grouping id (binary)
    uint32_t* slot_of;       // [n] the row's key
    uint32_t* first;         // [limit] first row of each key
    uint32_t* gid_of_slot;   // [limit]
    uint32_t* found;         // [kGbSort] the keys that occur, in any order
    unsigned long long* count;  // keys that occur
    uint32_t* many;          // count may be too small, but above kGbSort
    uint32_t* over;          // a key did not fit
    uint32_t limit;
    int check;               // AN inputs: report corrupt codes
    ErrList terr, gerr;
};

// MANY: beyond kGbSort groups, which the compaction counts, a new one is not added.
template <bool TENC, bool MANY>
AHEAD_DEV uint32_t small_gb_row(const SmallGb& g, uint64_t row, uint64_t tv, uint64_t gv) {
    const uint64_t t = TENC ? mulw(tv, g.k.tail.ainv, g.k.tail.width) : tv;
    if (TENC && t > g.k.tail.umax) g.terr.add(row);
    uint64_t key = t & g.k.keymask;
    if (g.k.binary) {
        const uint64_t gd = gv * g.k.gainv;
        if (g.check && gd > g.gmax) g.gerr.add(row);
        key = ((t & g.k.lmask) * (g.k.ngroups & g.k.lmask) + (gd & g.k.lmask)) & g.k.lmask;
    }
    if (key >= g.limit) {
        *g.over = 1;
        return 0;
    }
    const uint32_t s = (uint32_t)key, r = (uint32_t)row;
    if (r < ld_ca(g.first + s) && r < *(volatile uint32_t*)(g.first + s) && atomicMin(&g.first[s], r) == kNoRow &&
        (!MANY || ld_ca((const uint32_t*)g.count) <= kGbSort)) {
        const unsigned long long i = atomicAdd(g.count, 1ull);
        if (i < kGbSort) g.found[i] = s;
    }
    return s;
}

// The first rows, by one block in rounds: the keys that repeat are all in the
// table before the grid starts.
template <bool TENC>
__global__ void __launch_bounds__(1024) small_gb_seed_kernel(SmallGb g) {
    const uint64_t m = g.n < kGbSeedRows ? g.n : kGbSeedRows;
    for (uint64_t i = threadIdx.x; i < m; i += blockDim.x) {
        if (*(volatile uint32_t*)g.over) return;
        g.slot_of[i] = small_gb_row<TENC, false>(g, i, load_at(g.k.tail, i), g.k.binary ? load_at(g.k.grp, i) : 0);
    }
}

// Four consecutive rows per thread and step (their loads in flight together;
// 16-byte loads where the columns are aligned).
template <int W>
AHEAD_DEV void load4(const DCol& c, uint64_t i, bool vec, uint64_t (&v)[4]) {
    if (c.type != AHEAD_VOID && vec) {
        if constexpr (W == 8) {
            const ulonglong2* q = reinterpret_cast<const ulonglong2*>((const char*)c.data + i * 8);
            const ulonglong2 a = __ldg(q), b = __ldg(q + 1);
            v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
            return;
        } else if constexpr (W == 4) {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>((const char*)c.data + i * 4));
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            return;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = load_at(c, i + q);
}

// Rows from kGbSeedRows on, four per thread and step.
template <int TW, int GW, bool TENC, bool MANY>
AHEAD_DEV void small_gb_rows(const SmallGb& g, bool vec) {
    const uint64_t r0 = kGbSeedRows, m = (g.n - r0) / 4, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += stride) {
        const uint64_t row = r0 + 4 * i;
        uint64_t t[4], gv[4] = {0, 0, 0, 0};
        load4<TW>(g.k.tail, row, vec, t);
        if constexpr (GW) load4<GW>(g.k.grp, row, vec, gv);
        uint32_t s[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = small_gb_row<TENC, MANY>(g, row + q, t[q], gv[q]);
        *reinterpret_cast<uint4*>(g.slot_of + row) = make_uint4(s[0], s[1], s[2], s[3]);
    }
    if (blockIdx.x == 0 && threadIdx.x < (g.n - r0) % 4) {
        const uint64_t row = r0 + 4 * m + threadIdx.x;
        g.slot_of[row] = small_gb_row<TENC, MANY>(g, row, load_at(g.k.tail, row), GW ? load_at(g.k.grp, row) : 0);
    }
}

// TW, GW: the tail's and the grouping's width (GW 0: unary).  Where a quarter of the
// seed rows opened a group, most rows may: 1M groups of 3M rows all counted on one
// word took 199 us, 39 with the adds skipped beyond kGbSort.  The look before each add
// is for such inputs alone: in the loop of all it cost 30M rows of 400 groups 55 us
// instead of 50.
template <int TW, int GW, bool TENC>
__global__ void __launch_bounds__(256, GW ? 6 : 8) small_gb_insert_kernel(SmallGb g, bool vec) {
    // (a seed row's key did not fit: the hash table has the call.  Through L1: nearly
    // 10,000 warps' reads of one word at L2 took 2 to 19 us)
    if (ld_ca(g.over)) return;
    if (ld_ca((const uint32_t*)g.count) > kGbSeedRows / 4) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *g.many = 1;
        small_gb_rows<TW, GW, TENC, true>(g, vec);
    } else {
        small_gb_rows<TW, GW, TENC, false>(g, vec);
    }
}

// One block ranks up to kGbSort groups by first row (bitonic in shared memory)
// and writes each group's first head; more groups are left to the compaction.
template <bool AN>
__global__ void __launch_bounds__(1024) small_gb_rank_kernel(SmallGb g, DCol head, int decode_head, uint64_t aoid,
                                                             void* firsts, uint64_t cap) {
    __shared__ uint64_t s_k[kGbSort];
    const unsigned long long c = *g.count;
    if (c > kGbSort || *g.over) return;
    uint32_t m = 1;
    while (m < c) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
        const uint32_t s = i < c ? g.found[i] : 0;
        s_k[i] = i < c ? ((uint64_t)g.first[s] << 32 | s) : ~0ull;
    }
    __syncthreads();
    sort_block(s_k, m);
    for (uint32_t i = threadIdx.x; i < c; i += blockDim.x) {
        const uint64_t x = s_k[i];
        g.gid_of_slot[(uint32_t)x] = i;
        if (i < cap) {
            const uint64_t h = load_at(head, x >> 32);
            if (AN) ((uint64_t*)firsts)[i] = (decode_head ? dec_if(head, h, head.ainv) : h) * aoid;
            else ((uint32_t*)firsts)[i] = (uint32_t)h;
        }
    }
}

// Every row's group id, four rows per thread and step (8 x 4 bytes read and
// written per row: bound by HBM).  SORTED: only when the rank kernel ranked the groups.
template <bool AN, bool SORTED>
__global__ void __launch_bounds__(256) small_gb_assign_kernel(SmallGb g, uint64_t aoid, int binary, void* gids,
                                                              uint64_t cap) {
    if (SORTED && (*g.count > kGbSort || *g.over)) return;
    const uint64_t n = g.n < cap ? g.n : cap, m = n / 4, stride = (uint64_t)gridDim.x * blockDim.x;
    auto gid = [&](uint64_t row, uint32_t s) -> uint64_t {
        const uint32_t id = g.gid_of_slot[s];
        if (!AN) return id;
        const uint64_t v = (uint64_t)id * aoid;
        // (the binary dictionary keeps the code in an oid_t: see gb_assign_kernel)
        return (binary && (v >> 32) && g.first[s] != (uint32_t)row) ? (uint64_t)(uint32_t)v : v;
    };
    const bool vec = ((uintptr_t)gids & 15) == 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += stride) {
        const uint4 s = *reinterpret_cast<const uint4*>(g.slot_of + 4 * i);
        const uint64_t v[4] = {gid(4 * i, s.x), gid(4 * i + 1, s.y), gid(4 * i + 2, s.z), gid(4 * i + 3, s.w)};
        if (AN && vec) {
            ulonglong2* o = reinterpret_cast<ulonglong2*>((uint64_t*)gids + 4 * i);
            o[0] = make_ulonglong2(v[0], v[1]);
            o[1] = make_ulonglong2(v[2], v[3]);
        } else if (!AN && vec) {
            reinterpret_cast<uint4*>(gids)[i] = make_uint4((uint32_t)v[0], (uint32_t)v[1], (uint32_t)v[2],
                                                           (uint32_t)v[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) store_at(gids, AN ? 8 : 4, 4 * i + q, v[q]);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < n % 4) {
        const uint64_t row = 4 * m + threadIdx.x;
        store_at(gids, AN ? 8 : 4, row, gid(row, g.slot_of[row]));
    }
}

inline uint32_t gb_limit(uint64_t n) {
    uint64_t l = kGbMinLimit;
    while (l < 2 * n && l < kGbMaxLimit) l <<= 1;
    return (uint32_t)l;
}

inline size_t small_gb_scratch(uint64_t n) {
    return (size_t)gb_limit(n) * 8 + n * 4 + kGbSort * 4 + 2 * kErrListBytes + 4096;
}

// Counters 10-14 of the call: groups, `over`, corrupt tails, corrupt grouping codes, `many`.
constexpr int kGbCount = 10, kGbOver = 11, kGbTail = 12, kGbGrp = 13, kGbMany = 14, kGbCounters = 15;

// The group-by through the first-row table: everything up to the group ids of
// up to kGbSort groups.
template <bool AN>
SmallGb launch_small_gb(OpScope& s, const GbKey& k, uint64_t n, uint64_t gmax, const DCol& head, int decode_head,
                        uint64_t aoid, ahead_bat* gids, ahead_bat* firsts, uint64_t cap) {
    cudaStream_t st = s.ctx->stream;
    SmallGb g;
    g.k = k;
    g.n = n;
    g.gmax = gmax;
    g.limit = gb_limit(n);
    g.first = (uint32_t*)s.alloc((size_t)g.limit * 4);
    g.gid_of_slot = (uint32_t*)s.alloc((size_t)g.limit * 4);
    g.slot_of = (uint32_t*)s.alloc(n * 4);
    g.found = (uint32_t*)s.alloc(kGbSort * 4);
    g.count = (unsigned long long*)(s.d_counters + kGbCount);
    g.over = (uint32_t*)(s.d_counters + kGbOver);
    g.many = (uint32_t*)(s.d_counters + kGbMany);
    g.check = AN;
    g.terr = err_list(s, kGbTail);
    g.gerr = err_list(s, kGbGrp);
    cudaMemsetAsync(g.first, 0xff, (size_t)g.limit * 4, st);
    const bool vec = ((uintptr_t)k.tail.data & 15) == 0 && (!k.binary || ((uintptr_t)k.grp.data & 15) == 0);
    small_gb_seed_kernel<AN><<<1, 1024, 0, st>>>(g);
    s.launched();
    if (n > kGbSeedRows) {
        const uint32_t blocks = grid_for((n - kGbSeedRows + 3) / 4, 256);
        const uint32_t grid = blocks < (uint32_t)s.ctx->num_sms * 8 ? blocks : (uint32_t)s.ctx->num_sms * 8;
        by_width(k.tail.width, [&](auto tag) -> int {
            constexpr int TW = decltype(tag)::value;
            if (k.binary) small_gb_insert_kernel<TW, AN ? 8 : 4, AN><<<grid, 256, 0, st>>>(g, vec);
            else small_gb_insert_kernel<TW, 0, AN><<<grid, 256, 0, st>>>(g, vec);
            return 0;
        });
        s.launched();
    }
    small_gb_rank_kernel<AN><<<1, 1024, 0, st>>>(g, head, decode_head, aoid, firsts->tail.data,
                                                 firsts->tail.data ? cap : 0);
    s.launched();
    if (gids->tail.data) {
        small_gb_assign_kernel<AN, true><<<grid_for((n + 3) / 4, 256), 256, 0, st>>>(g, aoid, k.binary,
                                                                                     gids->tail.data, cap);
        s.launched();
    }
    return g;
}

// Grouped sums: sum[gid] += t * (AResult * AT^-1) over rows with a valid
// group id (aggregateAN.tcc:92-111), and the rows of corrupt codes listed on the
// way (see ErrList).  Up to kPrivWords groups add in shared memory: an entry is
// two 32-bit words, the low one's carry going into the high one (a 64-bit add
// there is a loop of compare-and-swaps), and few groups get a copy per lane or
// some lanes, so that lanes with the same group do not queue for one word.  Two
// neighbouring rows per thread, four such pairs in flight (two, in 40 registers,
// took 54 us).  12M (resbigint, 280 groups): 47 us (192 MB, 4.1 TB/s), both columns
// checked; before, 75, and 28 for the checks of each column.
constexpr uint32_t kPrivWords = 4096;

struct GroupSum {
    const char *tail, *grp;
    uint64_t n, tinv, tmax, ginv, gmax, ngroups, enc;
    unsigned long long* sums;
    uint32_t copies, tail_check;  // copies: a power of two up to 32; 0: adds in global memory
    ErrList terr, gerr;
};

template <int WT, int WG, bool CHECK>
__global__ void __launch_bounds__(256, 4) grouped_sum_kernel(GroupSum a) {
    constexpr int U = 4;
    __shared__ uint32_t s_lo[kPrivWords], s_hi[kPrivWords];
    const uint32_t C = a.copies, mine = threadIdx.x & (C - 1), used = (uint32_t)a.ngroups * C;
    if (C) {
        for (uint32_t i = threadIdx.x; i < used; i += blockDim.x) s_lo[i] = s_hi[i] = 0;
        __syncthreads();
    }
    const bool vt = (uintptr_t)a.tail % (2 * WT) == 0, vg = (uintptr_t)a.grp % (2 * WG) == 0;
    auto one = [&](uint64_t t, uint64_t g, uint64_t row) {
        const uint64_t gid = g * a.ginv;
        if (CHECK) {
            const bool bt = a.tail_check && mulw(t, a.tinv, WT) > a.tmax;
            if (bt || gid > a.gmax) {
                if (bt) a.terr.add(row);
                if (gid > a.gmax) a.gerr.add(row);
            }
        }
        if (gid > a.gmax || gid >= a.ngroups) return;
        const unsigned long long x = t * a.enc;
        if (C) {
            const uint32_t at = (uint32_t)gid * C + mine, lo = (uint32_t)x;
            const uint32_t hi = (uint32_t)(x >> 32) + (atomicAdd(&s_lo[at], lo) + lo < lo ? 1u : 0u);
            if (hi) atomicAdd(&s_hi[at], hi);
        } else {
            atomicAdd(&a.sums[gid], x);
        }
    };
    const uint64_t np = a.n / 2, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < np; p += U * stride) {
        uint64_t t[U][2], g[U][2];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (p + u * stride < np) {
                load_pair<WT>(a.tail, p + u * stride, vt, t[u]);
                load_pair<WG>(a.grp, p + u * stride, vg, g[u]);
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t q = p + u * stride;
            if (q >= np) break;
            one(t[u][0], g[u][0], 2 * q);
            one(t[u][1], g[u][1], 2 * q + 1);
        }
    }
    if ((a.n & 1) && blockIdx.x == 0 && threadIdx.x == 0)
        one(gmem_ld<WT>(a.tail, a.n - 1), gmem_ld<WG>(a.grp, a.n - 1), a.n - 1);
    if (C) {
        __syncthreads();
        for (uint32_t g = threadIdx.x; g < a.ngroups; g += blockDim.x) {
            unsigned long long x = 0;
            for (uint32_t c = 0; c < C; ++c) x += ((unsigned long long)s_hi[g * C + c] << 32) + s_lo[g * C + c];
            if (x) atomicAdd(&a.sums[g], x);
        }
    }
}

// The copies of each group's entry, and a grid of as many blocks as run at once
// (six an SM by shared memory) or as have 16 rows a thread.
inline uint32_t sum_copies(uint64_t ngroups) {
    uint32_t c = ngroups <= kPrivWords ? 1 : 0;
    while (c && c < 32 && ngroups * c * 2 <= kPrivWords) c *= 2;
    return c;
}
inline uint32_t sum_grid(const ahead_ctx* ctx, uint64_t n) {
    const uint64_t g = (n + 256 * 16 - 1) / (256 * 16), most = (uint64_t)ctx->num_sms * 6;
    return (uint32_t)(g < most ? (g ? g : 1) : most);
}

// hash<str_t>::get (miscellaneous.hpp:99-119): the Java-style string hash of
// a slot's chars up to its NUL (at most `width`), in 64 bits; each char is
// signed, and the multiplier's update (x 31) goes through a 32-bit int.
AHEAD_DEV uint64_t str_hash(const char* s, uint64_t width) {
    uint64_t len = 0;
    while (len < width && s[len]) ++len;
    uint64_t hash = 0, mult = 1;
    for (uint64_t k = len; k-- > 0;) {
        hash += (uint64_t)(int64_t)(signed char)s[k] * mult;
        const int32_t shifted = (int32_t)(uint32_t)(mult << 5);
        mult = (uint64_t)(int64_t)shifted - mult;
    }
    return hash;
}

// The binary group-by's keys over a string tail: hash(row) * numGroups + g
// in the larger type of v2_str_t, v2_bigint_t (groupbyAN.tcc:144).
__global__ void gb_insert_str_kernel(HashTab h, const char* strs, uint64_t width, DCol grp, uint64_t gainv,
                                     uint64_t ngroups, uint64_t n, uint32_t* slot_of, uint32_t* first) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t key = str_hash(strs + i * width, width) * ngroups + load_at(grp, i) * gainv;
        const uint32_t s = ht_insert(h, key);
        slot_of[i] = s;
        if ((uint32_t)i < first[s]) atomicMin(&first[s], (uint32_t)i);  // (a stale word is only larger)
    }
}

ahead_errvec* ev(ahead_errvec* errs, int k) { return errs ? &errs[k] : nullptr; }

int run_groupby(ahead_ctx* ctx, const ahead_bat* in, const ahead_bat* grouping, uint64_t ngroups, uint64_t aoid,
                uint64_t aoidinv, ahead_bat* gids, ahead_bat* firsts, uint64_t cap, ahead_errvec* errs, bool binary) {
    const int H = in->head.type, T = in->tail.type;
    const int eH = type_encoded(H);
    const uint64_t n = in->count;
    set_meta(&gids->head, AHEAD_VOID, 1, 1, 0, 0);
    set_meta(&gids->tail, AHEAD_RESOID, aoid, aoidinv, kRes56Max, 0);
    set_meta(&firsts->head, AHEAD_VOID, 1, 1, 0, 0);
    set_meta(&firsts->tail, AHEAD_RESOID, aoid, aoidinv, kRes56Max, 0);
    if (errs) {
        ev_begin(&errs[0], eH);
        ev_begin(&errs[1], 1);
        if (binary) ev_begin(&errs[2], 1);
    }
    gids->count = n;
    firsts->count = 0;
    if (!n) return AHEAD_OK;
    GbKey k;
    k.tail = dcol(in->tail);
    k.grp = binary ? dcol(grouping->tail) : dcol(in->tail);
    k.keymask = wmask(type_base_width(T));
    k.lmask = wmask(type_width(type_larger_of(T)));
    k.ngroups = ngroups;
    k.gainv = binary ? grouping->tail.Ainv : 0;
    k.binary = binary;
    const DCol hc = dcol(in->head);
    OpScope s(ctx);
    auto check_head = [&] {
        if (eH) run_colcheck(s, in->head, n, hc.ainv, hc.umax, hc.width, aoid, ev(errs, 0), 1);
    };
    auto check_tail = [&] { run_colcheck(s, in->tail, n, k.tail.ainv, k.tail.umax, k.tail.width, aoid, ev(errs, 1), 2); };
    auto check_grp = [&] {
        run_colcheck(s, grouping->tail, n, grouping->tail.Ainv, grouping->tail.unenc_max, 8, aoid, ev(errs, 2), 3);
    };
    // the error vectors from the lists the insert pass filled, once the counters are read back
    auto settle = [&](const ErrList& terr, const ErrList& gerr) -> int {
        const bool ok_t = settle_err_list(s, terr, kGbTail, aoid, ev(errs, 1));
        const bool ok_g = !binary || settle_err_list(s, gerr, kGbGrp, aoid, ev(errs, 2));
        if (!ok_t || !ok_g) {  // a column with many corrupt codes
            int r = s.reserve(2 * colcheck_scratch(n));
            if (r) return r;
            if (!ok_t) check_tail();
            if (!ok_g) check_grp();
            r = s.finish(4);
            if (r) return r;
            if (errs && !ok_t) errs[1].count = s.counter(2);
            if (errs && !ok_g) errs[2].count = s.counter(3);
        }
        return s.wait();
    };
    auto first_op = [&](const uint32_t* slot_of, const uint32_t* first, uint32_t* gid_of_slot) {
        FirstOp op;
        op.base = (const char*)slot_of;
        op.first = first;
        op.gid_of_slot = gid_of_slot;
        op.head = hc;
        op.aoid = aoid;
        op.cap = firsts->tail.data ? cap : 0;
        op.firsts = (uint64_t*)firsts->tail.data;
        op.acc = nullptr;
        op.decode_head = binary;
        return op;
    };
    int rc = s.reserve(small_gb_scratch(n) + compact_scratch<FirstOp>(n) + (eH ? colcheck_scratch(n) : 0));
    if (rc) return rc;
    const SmallGb g = launch_small_gb<true>(s, k, n, binary ? grouping->tail.unenc_max : 0, hc, binary, aoid, gids,
                                            firsts, cap);
    check_head();
    rc = s.finish(kGbCounters);
    if (rc) return rc;
    if (!s.counter(kGbOver)) {
        uint64_t groups = s.counter(kGbCount);
        if (errs && eH) errs[0].count = s.counter(1);
        if (groups > kGbSort) {  // ranked by the compaction of the rows that are their key's first
            run_compact(s, first_op(g.slot_of, g.first, g.gid_of_slot), n, 0);
            if (gids->tail.data) {
                small_gb_assign_kernel<true, false><<<grid_for((n + 3) / 4, 256), 256, 0, ctx->stream>>>(
                    g, aoid, binary, gids->tail.data, cap);
                s.launched();
            }
            if (s.counter(kGbMany)) {
                rc = s.finish(1);  // (leaves the lists' counters as they were read)
                if (rc) return rc;
                groups = s.counter(0);
            }
        }
        firsts->count = groups;
        rc = settle(g.terr, g.gerr);
        if (rc) return rc;
        return (n > cap || groups > cap) ? AHEAD_CAPACITY : AHEAD_OK;
    }
    // keys beyond the first-row table: the hash table
    const uint32_t cap_slots = ht_capacity(n);
    rc = s.reserve((size_t)(cap_slots + 1) * (8 + 4 + 4) + n * 4 + compact_scratch<FirstOp>(n) +
                   3 * colcheck_scratch(n) + 2 * kErrListBytes + 4096);
    if (rc) return rc;
    cudaStream_t st = ctx->stream;
    const ErrList terr = err_list(s, kGbTail), gerr = err_list(s, kGbGrp);
    HashTab h{};
    h.mask = cap_slots - 1;
    h.keys = (uint64_t*)s.alloc((size_t)(cap_slots + 1) * 8);
    uint32_t* first = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
    uint32_t* gid_of_slot = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
    uint32_t* slot_of = (uint32_t*)s.alloc(n * 4);
    cudaMemsetAsync(h.keys, 0xff, (size_t)(cap_slots + 1) * 8, st);
    cudaMemsetAsync(first, 0xff, (size_t)(cap_slots + 1) * 4, st);
    launch_gb_insert<true>(s, h, k, n, binary ? grouping->tail.unenc_max : 0, slot_of, first, terr, gerr);
    run_compact(s, first_op(slot_of, first, gid_of_slot), n, 0);
    if (gids->tail.data)
        gb_assign_kernel<<<grid_for(n, 256), 256, 0, st>>>(slot_of, first, gid_of_slot, n, aoid, binary,
                                                            (uint64_t*)gids->tail.data, cap);
    s.launched(2);
    check_head();
    rc = s.finish(kGbCounters);
    if (rc) return rc;
    firsts->count = s.counter(0);
    if (errs && eH) errs[0].count = s.counter(1);
    rc = settle(terr, gerr);
    if (rc) return rc;
    return (n > cap || firsts->count > cap) ? AHEAD_CAPACITY : AHEAD_OK;
}

bool head_ok(int h) { return h == AHEAD_VOID || h == AHEAD_OID || h == AHEAD_RESOID; }

// ------------------------------------------------------------ unencoded twins
// groupby (Normal/groupby.tcc:51-150): the same first-occurrence numbering on
// the raw tail (unary) or on t * numGroups + g in the tail's larger type
// (binary); outputs are oid_t: the group id of every row and the head of
// each group's first row.
struct FirstPlainOp {
    static constexpr int W = 4;
    static constexpr int NCH = 1;
    static constexpr bool ACC = false;
    static constexpr bool GATHER = true;
    static constexpr bool EMIT_V = false;
    static constexpr int NOUT = 1;
    const char* base;
    const uint32_t* first;
    uint32_t* gid_of_slot;
    DCol head;
    uint64_t cap;
    uint32_t* firsts;
    uint64_t* acc;
    AHEAD_DEV uint32_t eval(uint64_t v, uint64_t row, uint64_t&) const { return first[v] == (uint32_t)row ? 1u : 0u; }
    AHEAD_DEV uint64_t out0(int, uint64_t, uint64_t row) const { return row; }
    AHEAD_DEV uint64_t cap0() const { return ~0ull; }  // (every group gets its id)
    AHEAD_DEV void put0(int, uint64_t pos, uint64_t row) const {
        const uint32_t s = ((const uint32_t*)base)[row];
        gid_of_slot[s] = (uint32_t)pos;
        if (pos < cap) firsts[pos] = (uint32_t)load_at(head, row);
    }
};

__global__ void gb_assign_plain_kernel(const uint32_t* slot_of, const uint32_t* gid_of_slot, uint64_t n,
                                       uint32_t* gids, uint64_t cap) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n && i < cap;
         i += (uint64_t)gridDim.x * blockDim.x)
        gids[i] = gid_of_slot[slot_of[i]];
}

bool plain_groupable(int t) {
    return t == AHEAD_OID || t == AHEAD_TINYINT || t == AHEAD_SHORTINT || t == AHEAD_INT || t == AHEAD_RESOID ||
           t == AHEAD_RESTINY || t == AHEAD_RESSHORT || t == AHEAD_RESINT;
}

int run_groupby_plain(ahead_ctx* ctx, const ahead_bat* in, const ahead_bat* grouping, uint64_t ngroups,
                      ahead_bat* gids, ahead_bat* firsts, uint64_t cap, bool binary) {
    const int T = in->tail.type;
    const uint64_t n = in->count;
    default_meta(&gids->head, AHEAD_VOID);
    default_meta(&gids->tail, AHEAD_OID);
    default_meta(&firsts->head, AHEAD_VOID);
    default_meta(&firsts->tail, AHEAD_OID);
    gids->count = n;
    firsts->count = 0;
    if (!n) return AHEAD_OK;
    GbKey k;
    k.tail = dcol(in->tail);
    k.tail.enc = 0;  // the raw tail: an encoded tail is grouped by its codes
    k.grp = binary ? dcol(grouping->tail) : dcol(in->tail);
    k.keymask = wmask(type_width(T));
    k.lmask = wmask(type_width(type_larger_of(T)));
    k.ngroups = ngroups;
    k.gainv = 1;
    k.binary = binary;
    OpScope s(ctx);
    auto first_op = [&](const uint32_t* slot_of, const uint32_t* first, uint32_t* gid_of_slot) {
        FirstPlainOp op;
        op.base = (const char*)slot_of;
        op.first = first;
        op.gid_of_slot = gid_of_slot;
        op.head = dcol(in->head);
        op.cap = firsts->tail.data ? cap : 0;
        op.firsts = (uint32_t*)firsts->tail.data;
        op.acc = nullptr;
        return op;
    };
    int rc = s.reserve(small_gb_scratch(n) + compact_scratch<FirstPlainOp>(n));
    if (rc) return rc;
    const SmallGb g = launch_small_gb<false>(s, k, n, 0, dcol(in->head), 0, 1, gids, firsts, cap);
    rc = s.finish(kGbCounters);
    if (rc) return rc;
    if (!s.counter(kGbOver)) {
        uint64_t groups = s.counter(kGbCount);
        if (groups > kGbSort) {
            run_compact(s, first_op(g.slot_of, g.first, g.gid_of_slot), n, 0);
            if (gids->tail.data) {
                small_gb_assign_kernel<false, false><<<grid_for((n + 3) / 4, 256), 256, 0, ctx->stream>>>(
                    g, 1, binary, gids->tail.data, cap);
                s.launched();
            }
            rc = s.finish(1);
            if (rc) return rc;
            groups = s.counter(0);
        }
        firsts->count = groups;
        return (n > cap || groups > cap) ? AHEAD_CAPACITY : AHEAD_OK;
    }
    const uint32_t cap_slots = ht_capacity(n);
    rc = s.reserve((size_t)(cap_slots + 1) * (8 + 4 + 4) + n * 4 + compact_scratch<FirstPlainOp>(n) + 4096);
    if (rc) return rc;
    cudaStream_t st = ctx->stream;
    HashTab h{};
    h.mask = cap_slots - 1;
    h.keys = (uint64_t*)s.alloc((size_t)(cap_slots + 1) * 8);
    uint32_t* first = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
    uint32_t* gid_of_slot = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
    uint32_t* slot_of = (uint32_t*)s.alloc(n * 4);
    cudaMemsetAsync(h.keys, 0xff, (size_t)(cap_slots + 1) * 8, st);
    cudaMemsetAsync(first, 0xff, (size_t)(cap_slots + 1) * 4, st);
    launch_gb_insert<false>(s, h, k, n, 0, slot_of, first, ErrList{}, ErrList{});
    run_compact(s, first_op(slot_of, first, gid_of_slot), n, 0);
    if (gids->tail.data)
        gb_assign_plain_kernel<<<grid_for(n, 256), 256, 0, st>>>(slot_of, gid_of_slot, n, (uint32_t*)gids->tail.data,
                                                                  cap);
    s.launched(2);
    rc = s.finish(1);
    if (rc) return rc;
    firsts->count = s.counter(0);
    return (n > cap || firsts->count > cap) ? AHEAD_CAPACITY : AHEAD_OK;
}

// aggregate_sum<Result> (Normal/aggregate_scalar.tcc:47-58): the sum of the
// tails (the result type is at least as wide as the tail), mod 2^64 here and
// narrowed on the host.
__global__ void sum_plain_kernel(DCol tail, uint64_t n, unsigned long long* out) {
    unsigned long long acc = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        acc += load_at(tail, i);
    acc = warp_sum64(acc);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// arithmetic<Op, Result> (Normal/arithmetic_scalar.tcc:46-82) in the tails'
// width; division by zero yields 0 (undefined in the reference).
__global__ void arith_plain_kernel(DCol a, DCol b, uint64_t n, int op, int w, void* out) {
    const uint64_t m = wmask(w);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t x = load_at(a, i), y = load_at(b, i);
        uint64_t r;
        switch (op) {
            case AHEAD_ADD: r = x + y; break;
            case AHEAD_SUB: r = x - y; break;
            case AHEAD_MUL: r = x * y; break;
            default: r = y ? x / y : 0; break;
        }
        store_at(out, w, i, r & m);
    }
}

}  // namespace

extern "C" {

int ahead_gpu_groupby_an(ahead_ctx* ctx, const ahead_bat* in, uint64_t aoid, uint64_t aoidinv, ahead_bat* gids,
                         ahead_bat* firsts, uint64_t cap, ahead_errvec* errs) {
    if (!ctx || !in || !gids || !firsts) return AHEAD_BAD_ARG;
    if (!head_ok(in->head.type) || !type_encoded(in->tail.type))
        return fail(ctx, AHEAD_BAD_ARG, "groupbyAN: void/oid/resoid head and AN tail required");
    return run_groupby(ctx, in, nullptr, 0, aoid, aoidinv, gids, firsts, cap, errs, false);
}

int ahead_gpu_groupby2_an(ahead_ctx* ctx, const ahead_bat* in, const ahead_bat* grouping, uint64_t ngroups,
                          uint64_t aoid, uint64_t aoidinv, ahead_bat* gids, ahead_bat* firsts, uint64_t cap,
                          ahead_errvec* errs) {
    if (!ctx || !in || !grouping || !gids || !firsts) return AHEAD_BAD_ARG;
    if (!head_ok(in->head.type) || !type_encoded(in->tail.type) || grouping->head.type != AHEAD_VOID ||
        grouping->tail.type != AHEAD_RESOID)
        return fail(ctx, AHEAD_BAD_ARG, "groupbyAN: (void/oid/resoid, AN) and a (void, resoid) grouping required");
    if (in->count != grouping->count)
        return fail(ctx, AHEAD_SIZE_MISMATCH, "input BAT and existing grouping have different sizes!");
    return run_groupby(ctx, in, grouping, ngroups, aoid, aoidinv, gids, firsts, cap, errs, true);
}

int ahead_gpu_aggregate_sum_grouped_an(ahead_ctx* ctx, const ahead_bat* in, const ahead_bat* grouping,
                                       uint64_t ngroups, int result_type, uint64_t ar, uint64_t arinv, uint64_t aoid,
                                       ahead_bat* out, ahead_errvec* errs) {
    if (!ctx || !in || !grouping || !out) return AHEAD_BAD_ARG;
    const int H = in->head.type, T = in->tail.type;
    if (result_type != AHEAD_RESBIGINT) return fail(ctx, AHEAD_BAD_ARG, "aggregate_sum_groupedAN: resbigint result");
    if (!head_ok(H) || !(T == AHEAD_INT || T == AHEAD_RESINT || T == AHEAD_RESBIGINT || T == AHEAD_RESSHORT ||
                         T == AHEAD_RESTINY))
        return fail(ctx, AHEAD_BAD_ARG, "aggregate_sum_groupedAN: unsupported input types");
    if (grouping->head.type != AHEAD_VOID || grouping->tail.type != AHEAD_RESOID)
        return fail(ctx, AHEAD_BAD_ARG, "aggregate_sum_groupedAN: (void, resoid) grouping required");
    if (in->count != grouping->count) return fail(ctx, AHEAD_SIZE_MISMATCH, "bat and grouping must have the same size!");
    const int eH = type_encoded(H), eT = type_encoded(T);
    const int wh = type_width(type_encoded_of(H)), wt = type_width(type_encoded_of(T));
    const uint64_t AT = in->tail.A & wmask(wt);
    const uint64_t enc = ar * (eT ? inv_pow2(AT, 64) : 1ull);
    default_meta(&out->head, AHEAD_VOID);
    set_meta(&out->tail, AHEAD_RESBIGINT, ar, arinv, kRes56Max, 0);
    if (errs) {
        ev_begin(&errs[0], eH);
        ev_begin(&errs[1], eT);
        ev_begin(&errs[2], 1);
    }
    out->count = ngroups;
    const uint64_t n = in->count;
    OpScope s(ctx);
    int rc = s.reserve(3 * colcheck_scratch(n) + 2 * kErrListBytes);
    if (rc) return rc;
    if (ngroups && out->tail.data) cudaMemsetAsync(out->tail.data, 0, ngroups * 8, ctx->stream);
    auto check_tail = [&] { run_colcheck(s, in->tail, n, in->tail.Ainv & wmask(wt), in->tail.unenc_max & wmask(wt), wt, aoid, ev(errs, 1), 1); };
    auto check_grp = [&] { run_colcheck(s, grouping->tail, n, grouping->tail.Ainv, grouping->tail.unenc_max, 8, aoid, ev(errs, 2), 2); };
    GroupSum a;
    a.terr = err_list(s, 3);
    a.gerr = err_list(s, 4);
    const bool sum = n && out->tail.data;
    if (sum) {
        a.tail = (const char*)in->tail.data;
        a.grp = (const char*)grouping->tail.data;
        a.n = n;
        a.tinv = in->tail.Ainv & wmask(wt);
        a.tmax = in->tail.unenc_max & wmask(wt);
        a.tail_check = eT;
        a.ginv = grouping->tail.Ainv;
        a.gmax = grouping->tail.unenc_max;
        a.ngroups = ngroups;
        a.enc = enc;
        a.sums = (unsigned long long*)out->tail.data;
        a.copies = sum_copies(ngroups);
        by_width_enc(type_width(T), [&](auto tag) -> int {
            grouped_sum_kernel<decltype(tag)::value, 8, true><<<sum_grid(ctx, n), 256, 0, ctx->stream>>>(a);
            return 0;
        });
        s.launched();
    }
    if (n) {
        if (eH) run_colcheck(s, in->head, n, in->head.Ainv & wmask(wh), in->head.unenc_max & wmask(wh), wh, aoid, ev(errs, 0), 0);
        if (!sum && eT) check_tail();
        if (!sum) check_grp();
    }
    rc = s.finish(5);
    if (rc) return rc;
    if (errs && n) {
        if (eH) errs[0].count = s.counter(0);
        if (!sum) {
            if (eT) errs[1].count = s.counter(1);
            errs[2].count = s.counter(2);
        }
    }
    if (sum && errs) {
        const bool some = s.counter(3) + s.counter(4);
        const bool ok_t = !eT || settle_err_list(s, a.terr, 3, aoid, ev(errs, 1));
        const bool ok_g = settle_err_list(s, a.gerr, 4, aoid, ev(errs, 2));
        if (!ok_t || !ok_g) {  // a column with many corrupt codes
            rc = s.reserve(2 * colcheck_scratch(n));
            if (rc) return rc;
            if (!ok_t) check_tail();
            if (!ok_g) check_grp();
            rc = s.finish(3);
            if (rc) return rc;
            if (!ok_t) errs[1].count = s.counter(1);
            if (!ok_g) errs[2].count = s.counter(2);
        } else if (some) {
            return s.wait();
        }
    }
    return AHEAD_OK;
}


int ahead_gpu_groupby(ahead_ctx* ctx, const ahead_bat* in, ahead_bat* gids, ahead_bat* firsts, uint64_t cap) {
    if (!ctx || !in || !gids || !firsts) return AHEAD_BAD_ARG;
    if (!(in->head.type == AHEAD_VOID || in->head.type == AHEAD_OID) || !plain_groupable(in->tail.type))
        return fail(ctx, AHEAD_BAD_ARG, "groupby: void/oid head and an integer or code tail required");
    return run_groupby_plain(ctx, in, nullptr, 0, gids, firsts, cap, false);
}

int ahead_gpu_groupby2(ahead_ctx* ctx, const ahead_bat* in, const ahead_bat* grouping, uint64_t ngroups,
                       ahead_bat* gids, ahead_bat* firsts, uint64_t cap) {
    if (!ctx || !in || !grouping || !gids || !firsts) return AHEAD_BAD_ARG;
    if (!(in->head.type == AHEAD_VOID || in->head.type == AHEAD_OID) || !plain_groupable(in->tail.type) ||
        grouping->head.type != AHEAD_VOID || grouping->tail.type != AHEAD_OID)
        return fail(ctx, AHEAD_BAD_ARG, "groupby: (void/oid, integer) and a (void, oid) grouping required");
    if (in->count != grouping->count)
        return fail(ctx, AHEAD_SIZE_MISMATCH, "input BAT and existing grouping have different sizes!");
    return run_groupby_plain(ctx, in, grouping, ngroups, gids, firsts, cap, true);
}

int ahead_gpu_aggregate_sum_grouped(ahead_ctx* ctx, const ahead_bat* in, const ahead_bat* grouping,
                                    uint64_t ngroups, int result_type, ahead_bat* out) {
    if (!ctx || !in || !grouping || !out) return AHEAD_BAD_ARG;
    if (result_type != AHEAD_BIGINT || !(in->head.type == AHEAD_VOID || in->head.type == AHEAD_OID) ||
        in->tail.type != AHEAD_INT || grouping->head.type != AHEAD_VOID || grouping->tail.type != AHEAD_OID)
        return fail(ctx, AHEAD_BAD_ARG, "aggregate_sum_grouped: (void/oid, int), (void, oid) grouping, bigint result");
    if (in->count != grouping->count) return fail(ctx, AHEAD_SIZE_MISMATCH, "bat and grouping must have the same size!");
    default_meta(&out->head, AHEAD_VOID);
    default_meta(&out->tail, AHEAD_BIGINT);
    out->count = ngroups;
    const uint64_t n = in->count;
    OpScope s(ctx);
    int rc = s.reserve(0);
    if (rc) return rc;
    if (ngroups && out->tail.data) cudaMemsetAsync(out->tail.data, 0, ngroups * 8, ctx->stream);
    if (n && out->tail.data) {
        // group ids beyond numGroups index past the reference's vector; skipped here
        GroupSum a{};
        a.tail = (const char*)in->tail.data;
        a.grp = (const char*)grouping->tail.data;
        a.n = n;
        a.ginv = a.enc = 1;
        a.gmax = ~0ull;
        a.ngroups = ngroups;
        a.sums = (unsigned long long*)out->tail.data;
        a.copies = sum_copies(ngroups);
        grouped_sum_kernel<4, 4, false><<<sum_grid(ctx, n), 256, 0, ctx->stream>>>(a);
        s.launched();
    }
    return s.finish(0);
}

int ahead_gpu_aggregate_sum(ahead_ctx* ctx, const ahead_bat* in, int result_type, uint64_t* total) {
    if (!ctx || !in || !total) return AHEAD_BAD_ARG;
    const int T = in->tail.type;
    const bool ints = [](int t) {
        return t == AHEAD_TINYINT || t == AHEAD_SHORTINT || t == AHEAD_INT || t == AHEAD_BIGINT;
    }(T) && (result_type == AHEAD_TINYINT || result_type == AHEAD_SHORTINT || result_type == AHEAD_INT ||
             result_type == AHEAD_BIGINT);
    if (in->head.type != AHEAD_OID || !ints || type_width(result_type) < type_width(T))
        return fail(ctx, AHEAD_BAD_ARG, "aggregate_sum: (oid, integer) input and a result at least as wide");
    OpScope s(ctx);
    int rc = s.reserve(0);
    if (rc) return rc;
    if (in->count) {
        sum_plain_kernel<<<grid_for(in->count, 256), 256, 0, ctx->stream>>>(dcol(in->tail), in->count,
                                                                             (unsigned long long*)s.d_counters);
        s.launched();
    }
    rc = s.finish(1);
    if (rc) return rc;
    *total = (in->count ? s.counter(0) : 0) & wmask(type_width(result_type));
    return AHEAD_OK;
}

int ahead_gpu_arithmetic(ahead_ctx* ctx, int op, int result_type, const ahead_bat* a, const ahead_bat* b,
                         ahead_bat* out) {
    if (!ctx || !a || !b || !out) return AHEAD_BAD_ARG;
    const int T = a->tail.type;
    if (a->head.type != AHEAD_VOID || b->head.type != AHEAD_VOID || b->tail.type != T || result_type != T ||
        !(T == AHEAD_INT || T == AHEAD_RESINT) || op < AHEAD_ADD || op > AHEAD_DIV)
        return fail(ctx, AHEAD_BAD_ARG, "arithmetic: (void, int|resint) inputs of one type and that result type");
    if (a->count != b->count) return fail(ctx, AHEAD_SIZE_MISMATCH, "arithmetic: bat1->size() != bat2->size()");
    // the result keeps the first input's metadata (skeleton, miscellaneous.hpp:122-132)
    copy_meta(&out->head, AHEAD_VOID, &a->head);
    copy_meta(&out->tail, result_type, &a->tail);
    out->count = a->count;
    OpScope s(ctx);
    int rc = s.reserve(0);
    if (rc) return rc;
    if (a->count && out->tail.data) {
        arith_plain_kernel<<<grid_for(a->count, 256), 256, 0, ctx->stream>>>(dcol(a->tail), dcol(b->tail), a->count,
                                                                              op, type_width(T), out->tail.data);
        s.launched();
    }
    return s.finish(0);
}

int ahead_gpu_groupby2_str_an(ahead_ctx* ctx, const char* strs, uint64_t width, uint64_t count, uint64_t seqbase,
                              const ahead_bat* grouping, uint64_t ngroups, uint64_t aoid, uint64_t aoidinv,
                              ahead_bat* gids, ahead_bat* firsts, uint64_t cap, ahead_errvec* errs) {
    if (!ctx || !grouping || !gids || !firsts || !width || (count && !strs)) return AHEAD_BAD_ARG;
    if (grouping->head.type != AHEAD_VOID || grouping->tail.type != AHEAD_RESOID)
        return fail(ctx, AHEAD_BAD_ARG, "groupbyAN(str): (void, resoid) grouping required");
    if (count != grouping->count) return fail(ctx, AHEAD_SIZE_MISMATCH, "groupbyAN(str): sizes differ");
    set_meta(&gids->head, AHEAD_VOID, 1, 1, 0, 0);
    set_meta(&gids->tail, AHEAD_RESOID, aoid, aoidinv, kRes56Max, 0);
    set_meta(&firsts->head, AHEAD_VOID, 1, 1, 0, 0);
    set_meta(&firsts->tail, AHEAD_RESOID, aoid, aoidinv, kRes56Max, 0);
    if (errs) {
        ev_begin(&errs[0], 0);
        ev_begin(&errs[1], 0);
        ev_begin(&errs[2], 1);
    }
    const uint64_t n = count;
    gids->count = n;
    firsts->count = 0;
    OpScope s(ctx);
    const uint32_t cap_slots = ht_capacity(n);
    int rc = s.reserve((size_t)(cap_slots + 1) * (8 + 4 + 4) + n * 4 + compact_scratch<FirstOp>(n) +
                       colcheck_scratch(n) + 4096);
    if (rc) return rc;
    if (n) {
        cudaStream_t st = ctx->stream;
        HashTab h{};
        h.mask = cap_slots - 1;
        h.keys = (uint64_t*)s.alloc((size_t)(cap_slots + 1) * 8);
        uint32_t* first = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
        uint32_t* gid_of_slot = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
        uint32_t* slot_of = (uint32_t*)s.alloc(n * 4);
        cudaMemsetAsync(h.keys, 0xff, (size_t)(cap_slots + 1) * 8, st);
        cudaMemsetAsync(first, 0xff, (size_t)(cap_slots + 1) * 4, st);
        gb_insert_str_kernel<<<grid_for(n, 256), 256, 0, st>>>(h, strs, width, dcol(grouping->tail),
                                                               grouping->tail.Ainv, ngroups, n, slot_of, first);
        ahead_col vh{};
        vh.type = AHEAD_VOID;
        vh.seqbase = seqbase;
        FirstOp op;
        op.base = (const char*)slot_of;
        op.first = first;
        op.gid_of_slot = gid_of_slot;
        op.head = dcol(vh);
        op.aoid = aoid;
        op.cap = firsts->tail.data ? cap : 0;
        op.firsts = (uint64_t*)firsts->tail.data;
        op.acc = nullptr;
        op.decode_head = 1;
        run_compact(s, op, n, 0);
        if (gids->tail.data)
            gb_assign_kernel<<<grid_for(n, 256), 256, 0, st>>>(slot_of, first, gid_of_slot, n, aoid, 1,
                                                                (uint64_t*)gids->tail.data, cap);
        s.launched(2);
        run_colcheck(s, grouping->tail, n, grouping->tail.Ainv, grouping->tail.unenc_max, 8, aoid, ev(errs, 2), 1);
    }
    rc = s.finish(2);
    if (rc) return rc;
    firsts->count = n ? s.counter(0) : 0;
    if (errs && n) errs[2].count = s.counter(1);
    return (n > cap || firsts->count > cap) ? AHEAD_CAPACITY : AHEAD_OK;
}

int ahead_gpu_groupby2_str(ahead_ctx* ctx, const char* strs, uint64_t width, uint64_t count, uint64_t seqbase,
                           const ahead_bat* grouping, uint64_t ngroups, ahead_bat* gids, ahead_bat* firsts,
                           uint64_t cap) {
    if (!ctx || !grouping || !gids || !firsts || !width || (count && !strs)) return AHEAD_BAD_ARG;
    if (grouping->head.type != AHEAD_VOID || grouping->tail.type != AHEAD_OID)
        return fail(ctx, AHEAD_BAD_ARG, "groupby(str): (void, oid) grouping required");
    if (count != grouping->count) return fail(ctx, AHEAD_SIZE_MISMATCH, "groupby(str): sizes differ");
    default_meta(&gids->head, AHEAD_VOID);
    default_meta(&gids->tail, AHEAD_OID);
    default_meta(&firsts->head, AHEAD_VOID);
    default_meta(&firsts->tail, AHEAD_OID);
    const uint64_t n = count;
    gids->count = n;
    firsts->count = 0;
    OpScope s(ctx);
    const uint32_t cap_slots = ht_capacity(n);
    int rc = s.reserve((size_t)(cap_slots + 1) * (8 + 4 + 4) + n * 4 + compact_scratch<FirstPlainOp>(n) + 4096);
    if (rc) return rc;
    if (n) {
        cudaStream_t st = ctx->stream;
        HashTab h{};
        h.mask = cap_slots - 1;
        h.keys = (uint64_t*)s.alloc((size_t)(cap_slots + 1) * 8);
        uint32_t* first = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
        uint32_t* gid_of_slot = (uint32_t*)s.alloc((size_t)(cap_slots + 1) * 4);
        uint32_t* slot_of = (uint32_t*)s.alloc(n * 4);
        cudaMemsetAsync(h.keys, 0xff, (size_t)(cap_slots + 1) * 8, st);
        cudaMemsetAsync(first, 0xff, (size_t)(cap_slots + 1) * 4, st);
        gb_insert_str_kernel<<<grid_for(n, 256), 256, 0, st>>>(h, strs, width, dcol(grouping->tail), 1, ngroups, n,
                                                               slot_of, first);
        ahead_col vh{};
        vh.type = AHEAD_VOID;
        vh.seqbase = seqbase;
        FirstPlainOp op;
        op.base = (const char*)slot_of;
        op.first = first;
        op.gid_of_slot = gid_of_slot;
        op.head = dcol(vh);
        op.cap = firsts->tail.data ? cap : 0;
        op.firsts = (uint32_t*)firsts->tail.data;
        op.acc = nullptr;
        run_compact(s, op, n, 0);
        if (gids->tail.data)
            gb_assign_plain_kernel<<<grid_for(n, 256), 256, 0, st>>>(slot_of, gid_of_slot, n,
                                                                      (uint32_t*)gids->tail.data, cap);
        s.launched(2);
    }
    rc = s.finish(1);
    if (rc) return rc;
    firsts->count = n ? s.counter(0) : 0;
    return (n > cap || firsts->count > cap) ? AHEAD_CAPACITY : AHEAD_OK;
}

}  // extern "C"
