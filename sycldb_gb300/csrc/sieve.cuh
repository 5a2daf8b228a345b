// The sieve pass of the fused chain: any chain whose flags only shrink.
//
// The shape-specialised passes (namespace dense) are compiled for the op
// sequences of the common plans.  Every other chain used to go through the
// general interpreter (k_chain), which runs each op on all rows of a tile in
// turn, one dependent memory round trip after the other; small and plain ones
// still do (rows_from).  The sieve reads its ops at run
// time too, but orders its work as the specialised passes do: rows fall
// through three levels, each on full warps.
//
//   dense   the tests that read at most two columns (interval tests, column
//           comparisons, a join table small enough for a shared-memory bitmap,
//           one probe of a larger one) run on 8 rows per thread, the columns
//           copied a tile ahead into a shared-memory ring;
//   first   the survivors of a warp's 256 rows, listed in shared memory, run the
//           next op one row per lane;
//   second  the survivors of that, queued per warp as {row, join value}, run
//           the rest and the terminal whenever 32 are pending; every column
//           read from here on costs only the sectors that hold such rows.
//
// SSB flight 4.2 over 60 M rows (four joins, six columns, three keys): 1126 us
// in the general pass, 218 here.  What is left is the streaming of the two
// copied columns and the listing of the survivors first, then the probe of the
// customer table.
//
// Included by fused.cu (uses its namespace dense).
#pragma once

namespace sieve {

using dense::cp_async_wait;
using dense::kBitmapMax;
using dense::kDenseCap;

constexpr int kItems = 8;   // rows per thread and tile
constexpr int kQ = kItems / 4;
constexpr int kStages = 2;
constexpr int kStaged = 2;  // columns the ring holds: 32 KB, five blocks per SM
constexpr int kWarps = kThreads / 32;
constexpr int kMaxOps = SDB_CHAIN_MAX_OPS + 2;  // two more: full probes tested first and read for their value later

enum Kind { K_TEST = 0, K_CMP = 1, K_SEMI = 2, K_FULL = 3, K_BINOP = 4 };
enum { S_STAGED = 0, S_REG = 1, S_LIT = 2, S_COL = 3 };

struct Src {
    int32_t src;  // S_STAGED: ring slot idx on the dense level, the value listed with the row after it
    int32_t idx;  // slot or register
    int32_t lit;
    int32_t pad;
    const int32_t *col;
};

struct Op {
    int32_t kind, cmp, logic, bin;
    Src a, b;
    // K_TEST: (a - lo <= span | a - lo2 <= span2) != neg, unsigned
    uint32_t lo, span, lo2, span2, neg;
    int32_t kmin, kmax;  // probes: key range
    int32_t out_reg, ht_log2;
    int32_t bits;  // K_SEMI: the shared-memory bitmap holds the table's hits
    const void *ht;
};

struct Launch {
    uint64_t n;
    const uint8_t *flags_in;
    uint8_t *flags_out;
    const int32_t *slot[kStaged];
    int32_t nstaged, n_dense, n_ops;
    int32_t direct;   // no op after the dense ones drops a row: no second level
    int32_t listed;   // slot whose value a listed row keeps (S_STAGED after the dense level), -1: none
    int32_t first_reg;  // register the first level's op writes, -1: none
    Op ops[kMaxOps];
    Src value;
    uint64_t *sum_out;
    int32_t n_keys;
    Src keys[SDB_CHAIN_MAX_KEYS];
    int32_t key_min[SDB_CHAIN_MAX_KEYS];
    uint32_t mults[SDB_CHAIN_MAX_KEYS];
    uint64_t P;
    int32_t *out_keys[SDB_CHAIN_MAX_KEYS];
    uint64_t *out_sum;
    uint32_t *occ;
    const uint8_t *bitmap_ht;
    uint32_t bitmap_len;
    int32_t bitmap_kv;
};

// ---------------------------------------------------------------- dense level
struct Tile {
    const int4 *stage;  // this thread's rows: stage[slot * kThreads * kQ + q]
    uint64_t base;
    uint32_t valid, live;
};

__device__ __forceinline__ void fetch8(const Src &s, const Tile &T, int32_t (&v)[kItems])
{
    if (s.src == S_LIT) {
#pragma unroll
        for (int k = 0; k < kItems; k++) v[k] = s.lit;
        return;
    }
    if (s.src == S_STAGED) {
#pragma unroll
        for (int q = 0; q < kQ; q++) {
            const int4 x = T.stage[s.idx * kThreads * kQ + q];
            v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < kItems; k++) v[k] = (T.valid >> k) & 1u ? __ldcs(s.col + T.base + k) : 0;
}

__device__ __forceinline__ bool test(const Op &op, int32_t a)
{
    return ((((uint32_t)a - op.lo) <= op.span) | (((uint32_t)a - op.lo2) <= op.span2)) != (op.neg != 0);
}

__device__ __forceinline__ void dense_op(const Op &op, Tile &T, const uint32_t *s_bits)
{
    if (op.logic == SDB_AND && !__any_sync(0xffffffffu, T.live)) return;
    int32_t a[kItems];
    fetch8(op.a, T, a);
    uint32_t m = 0;
    if (op.kind == K_TEST) {
        const uint32_t lo = op.lo, lo2 = op.lo2, span = op.span, span2 = op.span2;
#pragma unroll
        for (int k = 0; k < kItems; k++)
            m |= (uint32_t)((((uint32_t)a[k] - lo) <= span) | (((uint32_t)a[k] - lo2) <= span2)) << k;
        if (op.neg) m ^= (1u << kItems) - 1u;
    } else if (op.kind == K_CMP) {
        int32_t b[kItems];
        fetch8(op.b, T, b);
#pragma unroll
        for (int k = 0; k < kItems; k++) m |= (uint32_t)sdb::compare(op.cmp, a[k], b[k]) << k;
    } else if (op.bits) {  // a probe on the bitmap: keys outside the table read word 0 and are masked off
        const int32_t kmin = op.kmin, kmax = op.kmax;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const uint32_t ok = dense::in_range(a[k], kmin, kmax);
            const uint32_t h = ok ? (uint32_t)a[k] - (uint32_t)kmin : 0u;
            m |= ((s_bits[h >> 5] >> (h & 31u)) & ok) << k;
        }
    } else {  // a probe of the live rows' entries, all eight reads in flight together
        const uint32_t kmin = (uint32_t)op.kmin, span = (uint32_t)op.kmax - kmin;
        int32_t e[kItems];
        if (op.kind == K_SEMI) {
            const uint8_t *ht = static_cast<const uint8_t *>(op.ht);
#pragma unroll
            for (int k = 0; k < kItems; k++) {
                const uint32_t h = (uint32_t)a[k] - kmin;
                e[k] = 0;
                if (((T.live >> k) & 1u) && h <= span) e[k] = __ldg(ht + h) != 0;
            }
        } else {
            const int2 *ht = static_cast<const int2 *>(op.ht);
#pragma unroll
            for (int k = 0; k < kItems; k++) {
                const uint32_t h = (uint32_t)a[k] - kmin;
                e[k] = 0;
                if (((T.live >> k) & 1u) && h <= span) e[k] = __ldg(&ht[h].x);
            }
        }
#pragma unroll
        for (int k = 0; k < kItems; k++) m |= (uint32_t)(e[k] == 1) << k;
    }
    T.live = sdb::logical4(op.logic, T.live, m) & T.valid;
}

// ---------------------------------------------------------------- row levels
// Registers are named members, chosen by selects: an array would go to local memory.
template <int NREGS>
struct Row {
    uint32_t row;
    int32_t listed;  // the listed slot's value
    int32_t r0, r1, r2, r3, r4, r5, r6, r7;  // the first NREGS in use
    bool live;
};

template <int NREGS>
__device__ __forceinline__ int32_t reg(const Row<NREGS> &R, int idx)
{
    int32_t v = R.r0;
    v = idx == 1 ? R.r1 : v;
    v = idx == 2 ? R.r2 : v;
    v = idx == 3 ? R.r3 : v;
    if constexpr (NREGS > 4) {
        v = idx == 4 ? R.r4 : v;
        v = idx == 5 ? R.r5 : v;
        v = idx == 6 ? R.r6 : v;
        v = idx == 7 ? R.r7 : v;
    }
    return v;
}

template <int NREGS>
__device__ __forceinline__ void set(Row<NREGS> &R, int idx, int32_t v)
{
    R.r0 = idx == 0 ? v : R.r0;
    R.r1 = idx == 1 ? v : R.r1;
    R.r2 = idx == 2 ? v : R.r2;
    R.r3 = idx == 3 ? v : R.r3;
    if constexpr (NREGS > 4) {
        R.r4 = idx == 4 ? v : R.r4;
        R.r5 = idx == 5 ? v : R.r5;
        R.r6 = idx == 6 ? v : R.r6;
        R.r7 = idx == 7 ? v : R.r7;
    }
}

template <int NREGS>
__device__ __forceinline__ void clear(Row<NREGS> &R)
{
    R.r0 = R.r1 = R.r2 = R.r3 = R.r4 = R.r5 = R.r6 = R.r7 = 0;
}

template <int NREGS>
__device__ __forceinline__ int32_t get(const Src &s, const Row<NREGS> &R)
{
    int32_t v = s.src == S_STAGED ? R.listed : s.lit;
    if (s.src == S_REG) v = reg(R, s.idx);
    if (s.src == S_COL) v = __ldg(s.col + R.row);
    return v;
}

template <int NREGS>
__device__ __forceinline__ void row_op(const Op &op, Row<NREGS> &R, const uint32_t *s_bits)
{
    if (!R.live) return;
    const int32_t a = get(op.a, R);
    switch (op.kind) {
    case K_TEST: R.live = test(op, a); break;
    case K_CMP: R.live = sdb::compare(op.cmp, a, get(op.b, R)); break;
    case K_SEMI: {
        const bool ok = dense::in_range(a, op.kmin, op.kmax);
        const uint32_t i = ok ? (uint32_t)a - (uint32_t)op.kmin : 0u;
        bool hit;
        if (op.bits) {
            hit = (s_bits[i >> 5] >> (i & 31u)) & 1u;
        } else if (op.ht_log2) {
            const uint32_t *w = static_cast<const uint32_t *>(op.ht);
            const int64_t s = ok ? sdb::oa_find<1>(w, op.ht_log2, sdb::oa_tag(a, op.kmin)) : -1;
            hit = s >= 0 && (__ldg(w + s) & 1u);
        } else {
            hit = ok && __ldg(static_cast<const uint8_t *>(op.ht) + i) != 0;
        }
        R.live = ok && hit;
        break;
    }
    case K_FULL: {
        const bool ok = dense::in_range(a, op.kmin, op.kmax);
        int2 e = make_int2(0, 0);
        if (op.ht_log2) {
            const int64_t s = ok ? sdb::oa_find<2>(static_cast<const uint32_t *>(op.ht), op.ht_log2, sdb::oa_tag(a, op.kmin)) : -1;
            if (s >= 0) {
                e = __ldg(static_cast<const int2 *>(op.ht) + s);
                e.x &= 1;
            }
        } else if (ok) {
            e = __ldg(static_cast<const int2 *>(op.ht) + ((uint32_t)a - (uint32_t)op.kmin));
        }
        R.live = e.x == 1;
        if (R.live) set(R, op.out_reg, e.y);
        break;
    }
    default: set(R, op.out_reg, sdb::binop(a, get(op.b, R), op.bin)); break;
    }
}

// The terminal for one row per lane.
template <int TERM, int NREGS>
__device__ __forceinline__ void finish(const Launch &L, const Row<NREGS> &R, uint32_t *s_key, uint32_t *s_sum, bool direct,
                                       uint64_t &acc)
{
    if (!R.live) return;
    const int32_t value = get(L.value, R);
    if (TERM == T_SUM) {
        acc += sdb::widen(value);
    } else {
        static_assert(SDB_CHAIN_MAX_KEYS == 4, "four keys by name");
        int32_t k0 = 0, k1 = 0, k2 = 0, k3 = 0;
        uint32_t h = 0;
        auto add = [&](int q, int32_t &k) {
            if (q >= L.n_keys) return;
            k = get(L.keys[q], R);
            h += ((uint32_t)k - (uint32_t)L.key_min[q]) * L.mults[q];
        };
        add(0, k0);
        add(1, k1);
        add(2, k2);
        add(3, k3);
        auto key_of = [k0, k1, k2, k3](auto q) {
            constexpr int i = decltype(q)::value;
            return i == 0 ? k0 : (i == 1 ? k1 : (i == 2 ? k2 : k3));
        };
        dense::group_row(L, s_key, s_sum, direct, h, value, L.n_keys, key_of);
    }
}

template <int TERM, int NREGS>
__global__ void __launch_bounds__(kThreads, TERM == T_FLAGS ? 6 : 5) k_sieve(const __grid_constant__ Launch L)
{
    extern __shared__ int4 s_buf[];  // [kStages][kStaged][kThreads][kQ], then the queues and the bitmap
    __shared__ uint32_t s_key[TERM == T_GROUP ? kDenseCap : 1];
    __shared__ uint32_t s_sum[TERM == T_GROUP ? 2 * kDenseCap : 1];
    __shared__ uint8_t s_list[TERM == T_FLAGS ? 1 : kThreads * kItems];  // per warp: offsets of its surviving rows
    __shared__ uint64_t s_part[kWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // per warp 64 second-level rows and, when the first level's op gives a
    // value, their values; then the bitmap
    uint32_t *s_queue = reinterpret_cast<uint32_t *>(s_buf + kStages * kStaged * kThreads * kQ);
    const uint32_t queue_words = TERM == T_FLAGS ? 0 : (L.first_reg >= 0 ? 128 : 64);
    uint32_t *s_bits = s_queue + kWarps * queue_words;
    constexpr uint64_t kTile = (uint64_t)kThreads * kItems;
    const uint64_t stride = (uint64_t)gridDim.x * kTile;
    uint64_t tile = (uint64_t)blockIdx.x * kTile;
    dense::issue_tile<kStages, kStaged, kItems>(L.slot, L.nstaged, L.n, s_buf, 0, tile);
    dense::group_table_reset<TERM>(s_key, s_sum);
    dense::stage_bitmap(L, s_bits);
    if (TERM == T_GROUP || L.bitmap_ht) __syncthreads();
    const bool direct_table = L.P <= kDenseCap;

    uint64_t acc = 0;
    uint32_t carried = 0;           // first-level rows kept from earlier tiles (warp-uniform), one per lane
    uint32_t c_row = 0;
    int32_t c_listed = 0;
    uint32_t queued = 0;            // second-level rows (warp-uniform)
    uint32_t *queue = s_queue + warp * queue_words;

    // One first-level group (`last`: the block's last, which empties the
    // queue).  One copy of the code serves every level's caller: the pass is large
    // enough to miss the instruction cache otherwise.
    auto group = [&](uint32_t row, int32_t listed, bool live, bool last) {
        Row<NREGS> R;
        R.row = row;
        R.listed = listed;
        R.live = live;
        clear(R);
        int from = L.n_dense;
        if (!L.direct) {
            row_op(L.ops[from], R, s_bits);
            const unsigned m = __ballot_sync(0xffffffffu, R.live);
            if (R.live) {
                const uint32_t at = queued + __popc(m & ((1u << lane) - 1u));
                queue[at] = R.row;
                if (L.first_reg >= 0) queue[64 + at] = (uint32_t)reg(R, L.first_reg);
            }
            queued += __popc(m);
            __syncwarp();
            from++;
        }
#pragma unroll 1
        do {
            if (!L.direct) {
                if (queued < (last ? 1u : 32u)) return;
                // the last (up to) 32 queued rows
                const uint32_t cnt = min(queued, 32u);
                queued -= cnt;
                R.live = lane < cnt;
                const uint32_t at = queued + (R.live ? lane : 0u);
                R.row = queue[at];
                clear(R);
                if (L.first_reg >= 0) set(R, L.first_reg, (int32_t)queue[64 + at]);
                __syncwarp();  // read before the queue grows again
            }
            bool any = true;
#pragma unroll 1
            for (int i = from; i < L.n_ops && any; i++) {
                row_op(L.ops[i], R, s_bits);
                any = __any_sync(0xffffffffu, R.live);
            }
            if (any) finish<TERM>(L, R, s_key, s_sum, direct_table, acc);
        } while (last && !L.direct);
    };

    int st = 0;
    bool last = false;  // one trip past the block's tiles takes what is left
    for (; !last; tile += stride, st ^= 1) {
        last = tile >= L.n;
        if (last && TERM == T_FLAGS) break;
        dense::issue_tile<kStages, kStaged, kItems>(L.slot, L.nstaged, L.n, s_buf, st ^ 1, tile + stride);
        cp_async_wait<1>();
        Tile T;
        T.stage = &s_buf[(st * kStaged * kThreads + threadIdx.x) * kQ];
        T.base = tile + (uint64_t)kItems * threadIdx.x;
        T.valid = (1u << kItems) - 1u;
        if (T.base + kItems > L.n) {  // (past the tiles: none)
            T.valid = 0;
#pragma unroll
            for (int k = 0; k < kItems; k++) T.valid |= (uint32_t)(T.base + k < L.n) << k;
        }
        T.live = T.valid;
        if (L.flags_in && T.valid) {
            uint32_t m = 0;
            if (T.valid == 0xffu && sdb::aligned(L.flags_in, 8)) {
                const uint64_t f = __ldcs(reinterpret_cast<const unsigned long long *>(L.flags_in + T.base));
#pragma unroll
                for (int k = 0; k < kItems; k++) m |= (uint32_t)(((f >> (8 * k)) & 0xffu) != 0) << k;
            } else {
#pragma unroll
                for (int k = 0; k < kItems; k++)
                    if ((T.valid >> k) & 1u) m |= (uint32_t)(L.flags_in[T.base + k] != 0) << k;
            }
            T.live = m;
        }
#pragma unroll 1
        for (int i = 0; i < L.n_dense; i++) dense_op(L.ops[i], T, s_bits);

        if constexpr (TERM == T_FLAGS) {
            if (T.valid == 0xffu && sdb::aligned(L.flags_out, 8)) {
                uint64_t f = 0;
#pragma unroll
                for (int k = 0; k < kItems; k++) f |= (uint64_t)((T.live >> k) & 1u) << (8 * k);
                *reinterpret_cast<uint64_t *>(L.flags_out + T.base) = f;
            } else {
#pragma unroll
                for (int k = 0; k < kItems; k++)
                    if ((T.valid >> k) & 1u) L.flags_out[T.base + k] = (uint8_t)((T.live >> k) & 1u);
            }
        } else {
            // the warp's surviving rows, in a list of offsets
            const uint32_t cnt = __popc(T.live);
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            uint8_t *list = s_list + warp * 32 * kItems;
            uint32_t pos = incl - cnt;
#pragma unroll
            for (int k = 0; k < kItems; k++)
                if ((T.live >> k) & 1u) list[pos++] = (uint8_t)(lane * kItems + k);
            __syncwarp();
            const uint32_t row0 = (uint32_t)(tile + (uint64_t)warp * 32 * kItems);
            const int32_t *ws = reinterpret_cast<const int32_t *>(&s_buf[(st * kStaged * kThreads + warp * 32) * kQ]) +
                                (L.listed > 0 ? L.listed : 0) * kThreads * kItems;
            const uint32_t avail = carried + total;
            uint32_t b = 0;
#pragma unroll 1
            for (; b + 32 <= avail || last; b += 32) {
                uint32_t row = c_row;
                int32_t v = c_listed;
                if (b + lane >= carried && !last) {  // else a carried row: only in the first group
                    const uint32_t r = list[b + lane - carried];
                    row = row0 + r;
                    v = L.listed >= 0 ? ws[r] : 0;
                }
                group(row, v, !last || lane < carried, last);
                if (last) break;
            }
            const uint32_t rem = last ? 0 : avail - b;
            if (lane < rem && b + lane >= carried) {
                const uint32_t r = list[b + lane - carried];
                c_row = row0 + r;
                c_listed = L.listed >= 0 ? ws[r] : 0;
            }
            carried = rem;
            __syncwarp();
        }
    }
    cp_async_wait<0>();
    if constexpr (TERM != T_FLAGS) {
        dense::block_flush<TERM>(L, s_key, s_sum, s_part, acc);
    }
}

// ---------------------------------------------------------------- host
// Rows from which a chain goes to the sieve, by its tests and probes.
// Below, the general pass: its threads hold 8 rows of a column each and
// sum or group them as they are, where the sieve lists every surviving row and
// takes 32 at a time through its levels -- less work when few survive, more
// when most do, and a tile of 2048 rows a block, too few of them on a small
// input.  us, general / sieve, where 1 in 100, a half and all rows pass each test:
//   SUM, a test          400 K  2.7/4.1  2.8/5.1  2.7/6.0    10 M  16/20  17/32  17/45
//   SUM, test and probe  1 M    7.8/8.3 (a half)             10 M  55/46 (a half), 48/30 (1 in 20)
//   SUM, two probes      1 M    11/8.6 (a half)              40 M  250/134
//   group-by, two probes 400 K  0.7 to 1 of the general pass; four 0.7 to 0.9
//   group-by, a test     400 K  7.5/6.4  9.6/10  8.3/12      40 M  178/67  210/189  204/303
//   flags, a test        1 M    3.0/3.1                      10 M  15/13
// A group-by whose P lies between the two passes' shared-memory tables
// overflows the sieve's (1000 groups, 10 M rows, half of them left: 112/180).
// Probes that give values alone may well drop nothing (a join with an unfiltered
// dimension; one of them, group-by, 40 M rows: 344/606).  A chain whose tests
// and semi joins drop nothing either is slower here, by up to a half (sums: up
// to twice).
inline uint64_t rows_from(const sdb_chain_desc &c, int term)
{
    if (term == T_FLAGS) return 1ull << 21;
    int tests = 0, semi = 0, full = 0;
    for (int i = 0; i < c.n_ops; i++) {
        const int k = c.ops[i].kind;
        tests += k == SDB_OP_SELECT || k == SDB_OP_SEARCH_RANGE || k == SDB_OP_SEARCH_POINTS;
        semi += k == SDB_OP_SEMI_PROBE;
        full += k == SDB_OP_FULL_PROBE;
    }
    if (tests + semi == 0) return ~0ull;
    if (semi + full >= 3) return 0;
    const bool between = term == T_GROUP && c.P > kDenseCap && c.P <= kCap;
    if (semi + full == 2) return term == T_GROUP && !between ? 1ull << 17 : 1ull << 20;
    if (term == T_GROUP) return between ? ~0ull : 1ull << 20;
    return tests && semi + full ? 1ull << 23 : ~0ull;
}

// Rows from which a bitmap of a table of so many bytes is packed: every block
// reads the whole table for it (200,000 key/value entries: 48 us, 16 as keys;
// 20,000: 6).  Without one its probe reads the table's entries: 10 M rows, half
// of them left by a test, group-by: 86 / 61 us with / without a bitmap of
// 200,000 entries, 47 / 59 of 20,000.
inline uint64_t bitmap_rows_from(uint64_t table_bytes) { return 64 * table_bytes; }

// Turns a checked chain into a sieve launch.  False: the chain is left to the
// general pass (a flag can come back after an op that is not a plain test of
// columns, a column is written, a register is written twice or read before it
// is written, nothing can run on the dense level, more than 2^31 rows, or an
// unaligned column).
inline bool convert(const ChainLaunch &C, int nregs, int term, Launch &D)
{
    const sdb_chain_desc &c = C.d;
    if (nregs > 8 || c.n >= (1ull << 31) || c.n == 0) return false;
    if (term != T_FLAGS && c.flags_out) return false;
    std::memset(&D, 0, sizeof D);
    D.n = c.n;
    D.flags_in = c.flags_in;
    D.flags_out = c.flags_out;
    D.listed = D.first_reg = -1;

    bool fill[SDB_CHAIN_MAX_REGS] = {}, written[SDB_CHAIN_MAX_REGS] = {};
    int32_t fill_lit[SDB_CHAIN_MAX_REGS] = {};
    auto src = [&](const sdb_operand &o, Src &s) {
        s = Src{};
        if (o.kind == SDB_SRC_COL) {
            s.src = S_COL;
            s.col = o.col;
        } else if (o.kind == SDB_SRC_LIT) {
            s.src = S_LIT;
            s.lit = o.lit;
        } else if (!written[o.reg]) {
            return false;
        } else if (fill[o.reg]) {
            s.src = S_LIT;
            s.lit = fill_lit[o.reg];
        } else {
            s.src = S_REG;
            s.idx = o.reg;
        }
        return true;
    };
    // a selection that starts the chain with NONE overwrites the input flags
    const bool fresh_start = c.n_ops > 0 && c.ops[0].logic_op == SDB_NONE &&
                             (c.ops[0].kind == SDB_OP_SELECT || c.ops[0].kind == SDB_OP_SEARCH_RANGE ||
                              c.ops[0].kind == SDB_OP_SEARCH_POINTS);
    if (fresh_start) D.flags_in = nullptr;
    std::vector<Op> ops;
    size_t fixed = 0;  // ops up to the last NONE or OR selection: they keep their order, on the dense level
    for (int i = 0; i < c.n_ops; i++) {
        const sdb_chain_op &o = c.ops[i];
        if (o.kind == SDB_OP_FILL) {
            if (o.out_col || written[o.out_reg]) return false;
            written[o.out_reg] = fill[o.out_reg] = true;
            fill_lit[o.out_reg] = o.a.lit;
            continue;
        }
        Op d{};
        if (!src(o.a, d.a)) return false;
        d.logic = SDB_AND;
        d.cmp = o.cmp_op;
        d.bin = o.bin_op;
        d.out_reg = -1;
        switch (o.kind) {
        case SDB_OP_SELECT:
        case SDB_OP_SEARCH_RANGE:
        case SDB_OP_SEARCH_POINTS: {
            d.logic = i == 0 && fresh_start ? (int)SDB_AND : o.logic_op;
            if (d.logic != SDB_NONE && d.logic != SDB_AND && d.logic != SDB_OR) return false;
            if (d.logic != SDB_AND) fixed = ops.size() + 1;
            sdb_operand lit = o.b;
            if (o.kind == SDB_OP_SELECT) {
                if (!src(o.b, d.b)) return false;
                if (d.b.src == S_LIT) {
                    lit.kind = SDB_SRC_LIT;
                    lit.lit = d.b.lit;
                }
            }
            RangeTest t{};
            if ((o.kind != SDB_OP_SELECT || d.b.src == S_LIT) && range_test(o.kind, o.cmp_op, lit.lit, o.lo, o.hi, t)) {
                d.kind = K_TEST;
                d.lo = (uint32_t)t.lo;
                d.lo2 = (uint32_t)t.lo2;
                d.span = t.span;
                d.span2 = t.span2;
                d.neg = (uint32_t)t.neg;
            } else if (o.kind == SDB_OP_SELECT) {
                d.kind = K_CMP;
            } else {
                return false;
            }
            break;
        }
        case SDB_OP_SEMI_PROBE:
        case SDB_OP_FULL_PROBE:
            d.kind = o.kind == SDB_OP_SEMI_PROBE ? K_SEMI : K_FULL;
            d.kmin = o.lo;
            d.kmax = o.hi;
            d.ht = o.ht;
            d.ht_log2 = o.ht_log2;
            if (o.kind == SDB_OP_FULL_PROBE) d.out_reg = o.out_reg;
            break;
        case SDB_OP_BINOP:
            if (!src(o.b, d.b)) return false;
            d.kind = K_BINOP;
            d.out_reg = o.out_reg;
            break;
        default: return false;
        }
        if (d.out_reg >= 0) {
            if (o.out_col || written[d.out_reg]) return false;
            written[d.out_reg] = true;
        }
        ops.push_back(d);
    }
    auto reads_reg = [](const Op &o) {
        return o.a.src == S_REG || ((o.kind == K_CMP || o.kind == K_BINOP) && o.b.src == S_REG);
    };
    auto plain = [&](const Op &o) { return (o.kind == K_TEST || o.kind == K_CMP) && !reads_reg(o); };
    for (size_t i = 0; i < fixed; i++)
        if (!plain(ops[i])) return false;

    // the ring: columns the dense level reads
    auto stage = [&](Src &s, int most) {
        if (s.src != S_COL) return true;
        for (int k = 0; k < D.nstaged; k++)
            if (D.slot[k] == s.col) {
                s.src = S_STAGED;
                s.idx = k;
                return true;
            }
        if (D.nstaged >= most || !sdb::aligned(s.col, 16)) return false;
        D.slot[D.nstaged] = s.col;
        s.src = S_STAGED;
        s.idx = D.nstaged++;
        return true;
    };
    std::vector<Op> run;
    std::vector<char> taken(ops.size(), 0);
    for (size_t i = 0; i < fixed; i++) {
        Op o = ops[i];
        stage(o.a, kStaged);
        if (o.kind == K_CMP) stage(o.b, kStaged);  // else read straight from the column
        run.push_back(o);
        taken[i] = 1;
    }
    // every op left only drops rows, so their order is free (registers
    // apart): tests of columns first, as many as two columns allow (all of them
    // when the flags are the result)
    for (size_t i = fixed; i < ops.size(); i++) {
        if (!plain(ops[i])) continue;
        Op o = ops[i];
        const int before = D.nstaged;
        const bool ok = stage(o.a, kStaged) && (o.kind != K_CMP || stage(o.b, kStaged));
        if (!ok && term != T_FLAGS) {
            D.nstaged = before;
            continue;
        }
        run.push_back(o);
        taken[i] = 1;
    }
    // then the probe with the smallest direct-address table that fits the
    // bitmap; a full probe still runs later, for its value
    int bit = -1;
    uint64_t best = ~0ull;
    for (size_t i = fixed; i < ops.size(); i++) {
        const Op &o = ops[i];
        if ((o.kind != K_SEMI && o.kind != K_FULL) || o.ht_log2 || o.a.src != S_COL) continue;
        const uint64_t len = o.kmin <= o.kmax ? (uint64_t)((int64_t)o.kmax - (int64_t)o.kmin + 1) : 0;
        if (len < 1 || len > kBitmapMax || len >= best || (o.kind == K_FULL && !sdb::aligned(o.ht, 16))) continue;
        if (c.n < bitmap_rows_from(len * (o.kind == K_FULL ? 8 : 1))) continue;
        best = len;
        bit = (int)i;
    }
    std::vector<size_t> again;  // full probes that still run for their value
    if (bit >= 0) {
        Op o = ops[bit];
        o.kind = K_SEMI;
        o.bits = 1;
        o.out_reg = -1;
        if (stage(o.a, kStaged)) {
            D.bitmap_ht = static_cast<const uint8_t *>(o.ht);
            D.bitmap_len = (uint32_t)best;
            D.bitmap_kv = ops[bit].kind == K_FULL;
            run.push_back(o);
            taken[bit] = 1;
            if (ops[bit].kind == K_FULL) again.push_back(bit);
        }
    }
    // and the first probe whose column the ring still has room for: eight rows
    // of a thread probe together, where one row per lane would wait for each
    // group of 32 in turn (flight 4.2, the customers of a fifth of the rows: the
    // plan's 339 us -> 278)
    if (!run.empty() && term != T_FLAGS)
        for (size_t i = fixed; i < ops.size(); i++) {
            if (taken[i] || (ops[i].kind != K_SEMI && ops[i].kind != K_FULL) || ops[i].ht_log2 || ops[i].a.src != S_COL ||
                ops[i].kmin > ops[i].kmax)
                continue;
            Op o = ops[i];
            o.out_reg = -1;
            if (!stage(o.a, kStaged)) continue;
            run.push_back(o);
            taken[i] = 1;
            if (ops[i].kind == K_FULL) again.push_back(i);
            break;
        }
    D.n_dense = (int)run.size();
    if (D.n_dense == 0 && !D.flags_in) return false;
    // the other filters in the plan's order, then what the last survivors
    // need: values of tables probed already, tests of registers, arithmetic
    for (size_t i = 0; i < ops.size(); i++)
        if (!taken[i] && !reads_reg(ops[i]) && ops[i].kind != K_BINOP) {
            run.push_back(ops[i]);
            taken[i] = 1;
        }
    bool drops = (int)run.size() > D.n_dense;
    for (size_t i : again) run.push_back(ops[i]);
    for (size_t i = 0; i < ops.size(); i++)
        if (!taken[i]) {
            run.push_back(ops[i]);
            drops |= ops[i].kind != K_BINOP;
        }
    if (run.size() > (size_t)kMaxOps) return false;
    D.n_ops = (int)run.size();
    D.direct = drops ? 0 : 1;
    if (term == T_FLAGS) {
        if (D.n_ops != D.n_dense) return false;
    } else {
        if (!src(c.value, D.value)) return false;
        D.n_keys = term == T_GROUP ? c.n_keys : 0;
        for (int q = 0; q < D.n_keys; q++) {
            if (!src(c.keys[q], D.keys[q])) return false;
            D.key_min[q] = c.key_min[q];
            D.mults[q] = C.mults[q];
            D.out_keys[q] = c.out_keys[q];
        }
        // a ring slot left over takes the column that the listed rows read next
        Src *next = D.n_ops > D.n_dense ? &run[D.n_dense].a : (D.n_keys ? &D.keys[0] : &D.value);
        if (stage(*next, kStaged)) D.listed = next->src == S_STAGED ? next->idx : -1;
        if (!D.direct) D.first_reg = run[D.n_dense].out_reg;
    }
    for (int i = 0; i < D.n_ops; i++) D.ops[i] = run[i];
    D.sum_out = c.sum_out;
    D.P = c.P;
    D.out_sum = c.out_sum;
    D.occ = c.occ;
    return true;
}

std::atomic<uint64_t> g_launches{0};  // read by sdb_sieve_launches

template <int TERM, int NREGS>
int launch(const Launch &D, cudaStream_t s)
{
    auto kern = k_sieve<TERM, NREGS>;
    constexpr int ring = kStages * kStaged * kThreads * kQ * (int)sizeof(int4);
    const int queues = TERM == T_FLAGS ? 0 : kWarps * (D.first_reg >= 0 ? 128 : 64) * 4;
    const int smem = ring + queues + (D.bitmap_ht ? (int)((D.bitmap_len + 31) / 32 * 4) : 0);
    static sdb::SmemLimit smem_limit;  // one per instantiation
    smem_limit.allow(ring + kWarps * 128 * 4 + (int)(kBitmapMax / 8), kern);  // (a launch it was refused for reports it)
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const uint64_t tile = (uint64_t)kThreads * kItems;
    const uint64_t blocks = std::min<uint64_t>((D.n + tile - 1) / tile, (uint64_t)num_sms() * per_sm);
    kern<<<(unsigned)blocks, kThreads, smem, s>>>(D);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return sdb_check_launch("sdb_fused_chain (sieve)");
}

// SDB_ERR_UNSUPPORTED (nothing launched) when the chain is left to the general
// pass: it is not the sieve's, or, unless `any_size`, the general pass is faster.
inline int dispatch(const ChainLaunch &C, int nregs, int term, bool any_size, cudaStream_t s)
{
    if (!any_size && C.d.n < rows_from(C.d, term)) return SDB_ERR_UNSUPPORTED;
    Launch D;
    if (!convert(C, nregs, term, D)) return SDB_ERR_UNSUPPORTED;
    if (term == T_FLAGS) return launch<T_FLAGS, 1>(D, s);
    if (term == T_SUM) return nregs <= 4 ? launch<T_SUM, 4>(D, s) : launch<T_SUM, 8>(D, s);
    return nregs <= 4 ? launch<T_GROUP, 4>(D, s) : launch<T_GROUP, 8>(D, s);
}

}  // namespace sieve
