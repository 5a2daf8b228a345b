// ORDER BY on the device: the stable order of row ids by a list of keys
// (int32 or uint64 columns, ascending or descending).
//
// The reference executor treats SORT as a pass-through (executor/
// ddor_executor.cpp:209-211); its unused host routine sort_table
// (kernels/sort.hpp:7-103) orders rows by the collation keys with std::sort,
// int32 keys compared as signed, aggregate (uint64) keys as unsigned.  This
// sort orders by the same comparisons; ties keep row order (stable), which
// std::sort does not promise.
//
// Up to kSmallSort rows: one launch that counts, for every row, the rows that
// come before it (k_sort_small).  Above: a least-significant-digit radix
// sort.  Each key becomes one or two 32-bit words whose unsigned order is the
// key's order (an int32 with its sign bit flipped, a uint64 as its low then
// its high word, every bit inverted for a descending key); the words are
// sorted 8 bits per pass from the last key's low word to the first key's high
// word, each pass moving (word, row id) pairs.  The digit counts of a word do
// not depend on the order of the rows, so one kernel takes all of them up
// front (k_sort_hist), a second turns them into first slots and drops the
// digits that are the same in every row (k_sort_plan: the high bytes of a
// year, of a group's sum), and a pass is then one kernel (k_sort_pass) that
// reads and writes each pair once.  Most sorts need only four of them: the
// first 32 bits of the keys laid end to end (each key less its smallest
// value, in the bits its range has) nearly always decide the order, so this
// head is sorted alone, and the few rows that tie in it are ordered afterwards
// (k_sort_range, k_sort_head, k_sort_ties).
#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace {

__device__ unsigned long long g_sort_errors;  // passes whose bounded look-back ran out

unsigned long long read_sort_errors(cudaStream_t s)
{
    unsigned long long v = 0, zero = 0;
    cudaMemcpyFromSymbolAsync(&v, g_sort_errors, sizeof v, 0, cudaMemcpyDeviceToHost, s);
    cudaMemcpyToSymbolAsync(g_sort_errors, &zero, sizeof zero, 0, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
    return v;
}
const int g_sort_reader = (sdb_errors_add_reader(&read_sort_errors), 0);

constexpr int kMaxKeys = 16;

struct SortKeys {
    const void *col[kMaxKeys];
    uint8_t wide[kMaxKeys];  // 1: uint64 column
    uint8_t desc[kMaxKeys];
    int n;
};

// Key k of a row as an unsigned value in the wanted order.
__device__ __forceinline__ uint64_t key_value(const SortKeys &K, int k, uint32_t row)
{
    if (K.wide[k]) {
        const uint64_t v = static_cast<const uint64_t *>(K.col[k])[row];
        return K.desc[k] ? ~v : v;
    }
    const uint32_t w = (uint32_t)static_cast<const int32_t *>(K.col[k])[row] ^ 0x80000000u;
    return K.desc[k] ? (uint32_t)~w : w;
}

// ---------------------------------------------------------------- small inputs
// A row's place is the number of rows that come before it.  A warp takes
// kSmallRows rows and walks all n rows, 32 at a time, comparing first keys
// held in registers; only a tie looks at the later keys.  n^2 comparisons,
// but no pass waits for another: latency at a few hundred rows, then issue.
// One launch: 37 rows by three keys 8.5 us (radix passes 136, the five
// launches per digit they had before 210).  The line lies where the two
// cross: 4096 rows by (int32, uint64) 42 against 115 us, by (year, sum), where
// one comparison in seven is a tie, 127 against 114; at 8192 rows 85 against
// 115 and 264 against 114.
constexpr uint32_t kSmallSort = 4096;
constexpr int kSmallRows = 4;
constexpr int kSmallThreads = 128;

// Columns to write in the order found, in place of the row ids: those of a
// result whose row count is still on the device.
struct SmallGather {
    const uint32_t *count;  // rows (NULL: no gather)
    uint32_t cap;           // nothing is ordered when there are more
    uint32_t *count_out;
    int ncols;
    const void *src[8];
    void *dst[8];
    uint8_t wide[8];
};

template <bool GATHER>
__global__ void __launch_bounds__(kSmallThreads) k_sort_small(const __grid_constant__ SortKeys K, uint32_t n,
                                                                uint32_t *__restrict__ perm,
                                                                const __grid_constant__ SmallGather G)
{
    if (GATHER) {
        n = *G.count;
        if (blockIdx.x == 0 && threadIdx.x == 0) *G.count_out = n;
        if (n > G.cap) return;
    }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t r0 = (blockIdx.x * (kSmallThreads / 32) + (threadIdx.x >> 5)) * kSmallRows;
    if (r0 >= n) return;  // warp-uniform
    uint64_t own[kSmallRows];
    uint32_t before[kSmallRows];
#pragma unroll
    for (int q = 0; q < kSmallRows; q++) {
        own[q] = key_value(K, 0, min(r0 + q, n - 1));
        before[q] = 0;
    }
    for (uint32_t j = lane; j < n; j += 32) {
        const uint64_t b = key_value(K, 0, j);
#pragma unroll
        for (int q = 0; q < kSmallRows; q++) {
            bool less = b < own[q];
            if (b == own[q]) {  // the later keys, then the row order
                const uint32_t i = min(r0 + q, n - 1);
                less = j < i;
                for (int k = 1; k < K.n; k++) {
                    const uint64_t x = key_value(K, k, i), y = key_value(K, k, j);
                    if (x != y) {
                        less = y < x;
                        break;
                    }
                }
            }
            before[q] += less;
        }
    }
#pragma unroll
    for (int q = 0; q < kSmallRows; q++) {
        const uint32_t at = __reduce_add_sync(0xffffffffu, before[q]);
        if (r0 + q >= n) break;
        if (!GATHER) {
            if (lane == 0) perm[at] = r0 + q;
        } else if (lane < (uint32_t)G.ncols) {
            if (G.wide[lane]) static_cast<uint64_t *>(G.dst[lane])[at] = static_cast<const uint64_t *>(G.src[lane])[r0 + q];
            else static_cast<int32_t *>(G.dst[lane])[at] = static_cast<const int32_t *>(G.src[lane])[r0 + q];
        }
    }
}

// ---------------------------------------------------------------- radix passes
constexpr int kSortThreads = 384;
constexpr int kSortItems = 16;                          // rows per thread
constexpr int kSortBlocks = 2;                          // resident per SM (80 registers a thread)
constexpr int kSortTile = kSortThreads * kSortItems;    // rows per block
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kFullPasses = kMaxKeys * 2 * 4;           // every digit of every key word
constexpr int kHeadPasses = 4;                          // the digits of the 32-bit head of the keys
constexpr int kMaxPasses = kFullPasses + kHeadPasses;

// What k_sort_plan decides for one digit pass.
struct PassPlan {
    uint32_t active;  // 0: not run (every row has the same digit, or the other way of sorting is taken)
    uint32_t first;   // starts from the row order itself
    uint32_t fresh;   // first active pass of its word: the words come from the key column
    uint32_t keep;    // the words are still needed after this pass
    uint32_t from;    // words are read from word[from] and written to word[1 - from]
    uint32_t to;      // row ids are read from perm[1 - to] and written to perm[to]
    uint32_t look;    // look-back words: this pass uses look[look] and clears look[1 - look]
    uint32_t pad;
};

struct SortState {
    uint32_t failed;               // a look-back ran out: the result is the identity
    uint32_t by_head;              // the rows are ordered by the head of their keys (and its tied runs)
    uint32_t head_exact;           // the head holds the whole keys: rows that tie are equal
    uint32_t head_ran;             // active passes of the head, if it was tried
    uint32_t ran;                  // active passes of the way taken
    uint32_t tile[kMaxPasses];     // next tile of each pass
    uint64_t not_min[kMaxKeys];    // ~ of each key's smallest value (so that zero is the start)
    uint64_t max[kMaxKeys];        // and its largest
    PassPlan plan[kMaxPasses];
    uint32_t count[kMaxPasses][256];  // digit counts, the head's last
    uint32_t slot[kMaxPasses][256];   // each digit's first slot
};

// The head of a row's keys: its keys less their smallest values, one after
// the other from the first key on, in as many bits as each key's range has,
// cut after `width` bits in all.  Unsigned order of heads is the order of the rows up
// to the cut.
struct Head {
    uint64_t min[kMaxKeys];
    int right[kMaxKeys], left[kMaxKeys];
    int keys;   // keys that give bits
    int bits;   // of the head
    int exact;  // no key is cut or left out
};

// Bits for n rows, in whole digits: enough that rows of evenly spread keys
// seldom tie (6 bits more than row ids have) up to 2^26 rows.  Above, a head that does not
// hold the whole keys ties too often (k_sort_plan): every digit is sorted.
__host__ __device__ inline int head_width(uint32_t n) { return n <= (1u << 18) ? 24 : 32; }

// Bits of the first k keys' ranges, at most `width`.
__device__ __forceinline__ int bits_of(const SortState *st, int k, int width)
{
    int bits = 0;
    for (int q = 0; q < k && bits < width; q++) bits += 64 - __clzll((long long)(st->max[q] + st->not_min[q] + 1));
    return bits;
}

// Smallest and largest value of key k (nothing when the keys before it fill
// the head).  Streams the column once.
constexpr int kHistThreads = 256;

__global__ void __launch_bounds__(kHistThreads) k_sort_range(const __grid_constant__ SortKeys K, int k, uint32_t n,
                                                               SortState *st)
{
    __shared__ uint64_t s_lo[kHistThreads / 32], s_hi[kHistThreads / 32];
    if (bits_of(st, k, head_width(n)) >= head_width(n)) return;
    uint64_t lo = ~0ull, hi = 0;
    const uint64_t stride = (uint64_t)gridDim.x * kHistThreads;
    uint64_t i = blockIdx.x * (uint64_t)kHistThreads + threadIdx.x;
    for (; i + 3 * stride < n; i += 4 * stride) {
        uint64_t v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = key_value(K, k, (uint32_t)(i + j * stride));
#pragma unroll
        for (int j = 0; j < 4; j++) {
            lo = min(lo, v[j]);
            hi = max(hi, v[j]);
        }
    }
    for (; i < n; i += stride) {
        const uint64_t v = key_value(K, k, (uint32_t)i);
        lo = min(lo, v);
        hi = max(hi, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31u) == 0) {
        s_lo[threadIdx.x >> 5] = lo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kHistThreads / 32; w++) {
            lo = min(lo, s_lo[w]);
            hi = max(hi, s_hi[w]);
        }
        atomicMax(reinterpret_cast<unsigned long long *>(&st->not_min[k]), (unsigned long long)~lo);
        atomicMax(reinterpret_cast<unsigned long long *>(&st->max[k]), (unsigned long long)hi);
    }
}

// Writes every row's head and counts its digits.  Bound by HBM: 16.8 M rows of
// an int32 and a uint64 key take 48 us (5.6 TB/s of keys and heads); with the
// key's width asked for at each of four rows 82.  A thread waits for eight
// rows of a key at once.
__global__ void __launch_bounds__(kHistThreads) k_sort_head(const __grid_constant__ SortKeys K, uint32_t n, SortState *st,
                                                              uint32_t *__restrict__ word)
{
    __shared__ uint32_t s_cnt[kHeadPasses][256];
    __shared__ Head s_head;
    for (uint32_t i = threadIdx.x; i < kHeadPasses * 256; i += kHistThreads) (&s_cnt[0][0])[i] = 0;
    if (threadIdx.x == 0) {
        const int width = head_width(n);
        int bits = 0, k = 0;
        bool cut = false;
        for (; k < K.n && bits < width; k++) {
            const int b = 64 - __clzll((long long)(st->max[k] + st->not_min[k] + 1));
            const int take = min(b, width - bits);
            s_head.min[k] = ~st->not_min[k];
            s_head.right[k] = b - take;
            s_head.left[k] = take;  // the shift, once every key has made room for the next
            cut |= take < b;
            bits += take;
        }
        int at = bits;
        for (int q = 0; q < k; q++) {
            at -= s_head.left[q];
            s_head.left[q] = at;
        }
        s_head.keys = k;
        s_head.bits = bits;
        s_head.exact = !cut && k == K.n;
        if (blockIdx.x == 0) st->head_exact = s_head.exact;
    }
    __syncthreads();
    const int digits = (s_head.bits + 7) / 8, keys = s_head.keys;
    constexpr int kItems = 8;
    const uint64_t stride = (uint64_t)gridDim.x * kHistThreads;
    for (uint64_t i0 = blockIdx.x * (uint64_t)kHistThreads + threadIdx.x; i0 < n; i0 += kItems * stride) {
        uint32_t h[kItems] = {};
        for (int k = 0; k < keys; k++) {
            const uint64_t least = s_head.min[k];
            const int right = s_head.right[k], left = s_head.left[k];
            if (K.wide[k]) {
                const uint64_t *col = static_cast<const uint64_t *>(K.col[k]), flip = K.desc[k] ? ~0ull : 0;
                uint64_t v[kItems];
#pragma unroll
                for (int j = 0; j < kItems; j++) v[j] = i0 + j * stride < n ? col[i0 + j * stride] ^ flip : least;
#pragma unroll
                for (int j = 0; j < kItems; j++) h[j] |= (uint32_t)((v[j] - least) >> right << left);
            } else {
                const uint32_t *col = static_cast<const uint32_t *>(K.col[k]), flip = K.desc[k] ? 0x7fffffffu : 0x80000000u;
                uint32_t v[kItems];
#pragma unroll
                for (int j = 0; j < kItems; j++) v[j] = i0 + j * stride < n ? col[i0 + j * stride] ^ flip : (uint32_t)least;
#pragma unroll
                for (int j = 0; j < kItems; j++) h[j] |= (uint32_t)((v[j] - least) >> right << left);
            }
        }
#pragma unroll
        for (int j = 0; j < kItems; j++) {
            if (i0 + j * stride >= n) break;
            word[i0 + j * stride] = h[j];
#pragma unroll
            for (int d = 0; d < kHeadPasses; d++)
                if (d < digits) atomicAdd(&s_cnt[d][(h[j] >> (8 * d)) & 255u], 1u);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kHeadPasses * 256; i += kHistThreads) {
        const uint32_t c = (&s_cnt[0][0])[i];
        if (c) atomicAdd(&st->count[kFullPasses + (i >> 8)][i & 255u], c);
    }
}

// Digit counts of every word of every key (blockIdx.y: the key; nothing when
// the rows are already ordered by the head).  A warp whose 32 rows share a digit
// adds them as one (the constant bytes of narrow ranges would serialise 32
// shared-memory atomics on one word).  Bound by those atomics, one per row
// and digit.
__global__ void __launch_bounds__(kHistThreads) k_sort_hist(const __grid_constant__ SortKeys K, uint32_t n, SortState *st)
{
    __shared__ uint32_t s_cnt[8][256];
    if (st->by_head) return;
    const int k = blockIdx.y;
    const int digits = K.wide[k] ? 8 : 4;
    int pass0 = 0;  // passes of the keys after this one run first
    for (int q = k + 1; q < K.n; q++) pass0 += K.wide[q] ? 8 : 4;
    for (uint32_t i = threadIdx.x; i < 8 * 256; i += kHistThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    constexpr int kItems = 4;
    // warp-uniform trips: the warp votes below need all 32 lanes
    for (uint64_t base = ((uint64_t)blockIdx.x * kHistThreads + (threadIdx.x & ~31u)) * kItems; base < n;
         base += (uint64_t)gridDim.x * kHistThreads * kItems) {
        uint64_t v[kItems];
#pragma unroll
        for (int j = 0; j < kItems; j++) {
            const uint64_t i = base + (uint64_t)j * 32 + lane;
            v[j] = i < n ? key_value(K, k, (uint32_t)i) : 0;
        }
#pragma unroll
        for (int j = 0; j < kItems; j++) {
            const uint64_t row = base + (uint64_t)j * 32;
            if (row >= n) break;
            const uint32_t here = (uint32_t)min((uint64_t)32, n - row);
#pragma unroll
            for (int d = 0; d < 8; d++) {
                if (d >= digits) break;
                const uint32_t x = (uint32_t)(v[j] >> (8 * d)) & 255u;
                const uint32_t x0 = __shfl_sync(0xffffffffu, x, 0);
                if (__all_sync(0xffffffffu, lane >= here || x == x0)) {
                    if (lane == 0) atomicAdd(&s_cnt[d][x], here);
                } else if (lane < here) {
                    atomicAdd(&s_cnt[d][x], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < (uint32_t)digits * 256; i += kHistThreads) {
        const uint32_t c = (&s_cnt[0][0])[i];
        if (c) atomicAdd(&st->count[pass0 + (i >> 8)][i & 255u], c);
    }
}

// Exclusive scan of 256 counts by the block's first 256 threads (every
// thread of the block calls it).
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t *s_warp)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31 && warp < 8) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8; w++) before += w < warp ? s_warp[w] : 0;
    __syncthreads();
    return x - v + before;
}

// One block: which passes run and each digit's first slot.  With `head` it
// looks at the head's digits: they are sorted when the head is the whole key,
// or when the counts say that at most one row in 64 should share its head with
// another (n times the product of the digits' collision probabilities); the
// few tied runs are ordered afterwards (k_sort_ties).  A tied run longer than
// kTieRows, possible when the digits depend on one another, sends the sort back to
// all digits of all words.
constexpr uint32_t kTieRows = 32;

__global__ void __launch_bounds__(256) k_sort_plan(SortState *st, int head, int passes, uint32_t n)
{
    __shared__ uint32_t s_warp[8];
    __shared__ float s_part[8];
    __shared__ PassPlan s_plan[kFullPasses];
    const uint32_t tried = st->head_ran;
    if (!head && st->by_head) return;
    const int p0 = head ? kFullPasses : 0;
    uint32_t ran = 0;
    float tied = (float)n;
    for (int p = 0; p < passes; p++) {
        const uint32_t c = st->count[p0 + p][threadIdx.x];
        // (a digit the head does not have was not counted)
        const bool active = __syncthreads_or(c != 0) && !__syncthreads_or(c == n);
        st->slot[p0 + p][threadIdx.x] = scan256(c, s_warp);
        if (head && active) {
            float x = (float)c / (float)n;
            x *= x;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if ((threadIdx.x & 31u) == 0) s_part[threadIdx.x >> 5] = x;
            __syncthreads();
            float t = 0;
            for (int w = 0; w < 8; w++) t += s_part[w];
            tied *= t;
        }
        if (threadIdx.x == 0) s_plan[p].active = active;
        ran += active;
    }
    if (threadIdx.x) return;
    const bool take = !head || st->head_exact || tied <= 1.0f / 64;
    uint32_t index = 0;
    int before = -1;  // the active pass before this one, of the same word
    for (int p = 0; p < passes; p++) {
        if ((p & 3) == 0) before = -1;
        PassPlan &q = s_plan[p];
        if (!take) q.active = 0;
        if (q.active) {
            q.first = index == 0;
            q.fresh = !head && before < 0;  // the head's words are in word[0]
            q.keep = head;                  // and k_sort_ties reads them sorted
            if (before >= 0) s_plan[before].keep = 1;
            q.from = index & 1u;
            q.to = (ran - 1u - index) & 1u;
            q.look = (tried + index) & 1u;
            q.pad = 0;
            before = p;
            index++;
        }
    }
    for (int p = 0; p < passes; p++) st->plan[p0 + p] = s_plan[p];
    st->ran = index;
    if (head) {
        st->by_head = take;
        st->head_ran = index;
    }
}

// Look-back words of (tile, digit): 0 = nothing yet, c + 1 = the tile holds c
// rows of the digit, kInclusive | c = it and all tiles before it hold c.
constexpr uint32_t kInclusive = 0x80000000u;
constexpr int kLookWindow = 8;        // earlier tiles read at a time
constexpr uint32_t kLookLimit = 1u << 20;  // polls before a look-back gives up, unless the caller says

struct PassArgs {
    const void *col;
    int32_t wide, hi, desc;
    int32_t pass;
    uint32_t n;
    uint32_t polls;       // of a look-back before it gives up
    SortState *st;
    uint32_t *look[2];    // [tiles][256] each
    uint32_t *perm[2];    // perm[0]: the caller's array, where the last active pass writes
    uint32_t *word[2];
};

__device__ __forceinline__ uint32_t key_word(const PassArgs &a, uint32_t row)
{
    uint32_t w;
    if (a.wide) {
        const uint64_t v = static_cast<const uint64_t *>(a.col)[row];
        w = a.hi ? (uint32_t)(v >> 32) : (uint32_t)v;
    } else {
        w = (uint32_t)static_cast<const int32_t *>(a.col)[row] ^ 0x80000000u;
    }
    return a.desc ? ~w : w;
}

__device__ __forceinline__ uint32_t load_look(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_look(uint32_t *p, uint32_t v)
{
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Rows of digit threadIdx.x in the tiles before `tile`: adds published counts
// backwards until one covers all earlier tiles.  ok = false when the wait
// ran out (after `limit` polls, or another tile's did).
__device__ __forceinline__ uint32_t look_back(const uint32_t *look, uint32_t tile, const uint32_t *failed, uint32_t limit,
                                              bool &ok)
{
    uint32_t before = 0, polls = 0;
    int64_t t = (int64_t)tile - 1;  // the latest tile not added yet
    while (limit) {
        uint32_t v[kLookWindow];
#pragma unroll
        for (int q = 0; q < kLookWindow; q++)
            v[q] = t >= q ? load_look(look + (size_t)(t - q) * 256 + threadIdx.x) : kInclusive;
        bool go = true;  // up to the first word not published yet: from there the window is read again
        bool done = false;
#pragma unroll
        for (int q = 0; q < kLookWindow; q++) {
            go = go && v[q] != 0;
            if (!go) continue;
            if (v[q] & kInclusive) {
                before += v[q] & ~kInclusive;
                done = true;
                go = false;
            } else {
                before += v[q] - 1u;
                t--;
            }
        }
        if (done) return before;
        if (++polls >= limit || ((polls & 1023u) == 0 && load_look(failed))) break;
    }
    ok = false;
    return before;
}

// Keeps in `peers` the lanes whose `bit` is zero or not as this lane's is: one
// bit of the ballot match of GPU multisplit (Ashkiani, Davidson, Meyer, Owens,
// 2016).  In PTX, so that the vote's predicate also turns the mask around; the
// same in C++ (peers &= bit ? m : ~m, or by a shifted-out mask) took 686 and 617
// us for a sort of 16.8 M rows by an int32 and a uint64 key, this 588.
__device__ __forceinline__ void keep_same_bit(unsigned &peers, uint32_t bit)
{
    asm volatile(
        "{ .reg .pred p; .reg .b32 m;\n"
        "  setp.ne.u32 p, %1, 0;\n"
        "  vote.sync.ballot.b32 m, p, 0xffffffff;\n"
        "  @!p not.b32 m, m;\n"
        "  and.b32 %0, %0, m; }\n"
        : "+r"(peers)
        : "r"(bit));
}

// One tile of a pass (FULL: all its rows exist).
template <bool FULL, int SHIFT>
__device__ __forceinline__ bool pass_tile(const PassArgs &a, const PassPlan &plan, uint32_t tile, uint32_t rows,
                                          uint2 *s_pair, uint32_t (*wc)[256], uint32_t *s_first,
                                          uint32_t *s_warp, uint32_t *s_stop)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t t0 = tile * (uint32_t)kSortTile;  // fits: at most 2^31 rows
    const uint32_t base = warp * (32u * kSortItems) + lane;
    auto valid = [&](int j) { return FULL || base + (uint32_t)j * 32 < rows; };
    uint32_t *look = a.look[plan.look];
    const uint32_t *perm_in = a.perm[plan.to ^ 1u] + t0 + base;

    uint32_t w[kSortItems], r[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; j++) {
        r[j] = t0 + base + (uint32_t)j * 32;
        if (!plan.first && valid(j)) r[j] = __ldcs(perm_in + j * 32);
    }
    if (plan.fresh) {
#pragma unroll
        for (int j = 0; j < kSortItems; j++) w[j] = valid(j) ? key_word(a, r[j]) : 0;
    } else {
        const uint32_t *word_in = a.word[plan.from] + t0 + base;
#pragma unroll
        for (int j = 0; j < kSortItems; j++) w[j] = valid(j) ? __ldcs(word_in + j * 32) : 0;
    }
    uint32_t rank[kSortItems / 2];  // two 16-bit ranks a word
#pragma unroll
    for (int j = 0; j < kSortItems; j++) {
        const uint32_t d = (w[j] >> SHIFT) & 255u;
        unsigned peers = FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, valid(j));
#pragma unroll
        for (int b = 0; b < 8; b++) keep_same_bit(peers, w[j] & (1u << (b + SHIFT)));
        // (lanes past the end get peers that are not theirs, and use nothing)
        const uint32_t below = __popc(peers & ((1u << lane) - 1u));
        const uint32_t had = wc[warp][d];
        if (j & 1) rank[j / 2] |= (had + below) << 16;
        else rank[j / 2] = had + below;
        __syncwarp();
        if (below == 0 && valid(j)) wc[warp][d] = had + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: the earlier warps' counts (in place), the tile's count, its
    // place in the tile
    uint32_t cnt = 0;
    if (threadIdx.x < 256) {
#pragma unroll
        for (int q = 0; q < kSortWarps; q++) {
            const uint32_t c = wc[q][threadIdx.x];
            wc[q][threadIdx.x] = cnt;
            cnt += c;
        }
        store_look(look + (size_t)tile * 256 + threadIdx.x, tile == 0 ? kInclusive | cnt : cnt + 1u);
    }
    const uint32_t tpre = scan256(cnt, s_warp);
    if (threadIdx.x < 256) {
#pragma unroll
        for (int q = 0; q < kSortWarps; q++) wc[q][threadIdx.x] += tpre;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; j++) {
        if (valid(j)) {
            const uint32_t d = (w[j] >> SHIFT) & 255u;
            const uint32_t at = wc[warp][d] + ((rank[j / 2] >> (16 * (j & 1))) & 0xffffu);
            s_pair[at] = make_uint2(w[j], r[j]);
        }
    }
    uint32_t before = 0;
    if (threadIdx.x < 256 && tile) {
        bool ok = true;
        before = look_back(look, tile, &a.st->failed, a.polls, ok);
        if (!ok) {
            store_look(&a.st->failed, 1u);
            *s_stop = 1;
        }
        store_look(look + (size_t)tile * 256 + threadIdx.x, kInclusive | (before + cnt));
    }
    if (threadIdx.x < 256) s_first[threadIdx.x] = a.st->slot[a.pass][threadIdx.x] + before - tpre;
    __syncthreads();
    if (*s_stop) return false;
    // out in tile order: slot p of digit d goes to s_first[d] + p
    uint32_t *perm_out = a.perm[plan.to], *word_out = a.word[plan.from ^ 1u];
    const bool keep = plan.keep;
    auto put = [&](uint32_t p) {
        const uint2 x = s_pair[p];
        const uint32_t at = s_first[(x.x >> SHIFT) & 255u] + p;
        if (keep) word_out[at] = x.x;
        perm_out[at] = x.y;
    };
    if (FULL) {
#pragma unroll 8
        for (int j = 0; j < kSortItems; j++) put(threadIdx.x + j * kSortThreads);
    } else {
        for (uint32_t p = threadIdx.x; p < rows; p += kSortThreads) put(p);
    }
    return true;
}

// Moves the (word, row id) pairs to their slots of one digit pass, stably; a
// block takes tiles of 6144 pairs until none is left.  Warp w owns the tile's
// pairs [512 w, 512 w + 512): their loads go out together, eight ballots per
// step of 32 give the lanes of one digit, a count per warp and digit carries
// the earlier steps.  The tile then publishes its
// digit counts, orders itself in shared memory, and meanwhile learns the
// counts of all earlier tiles from their published words (a word carries
// its own state, so no ordering of other memory is needed; tiles are handed
// out in order, so an earlier tile is always running or done).  It goes out
// in runs of equal digits.  A wait that runs out marks the sort failed and
// the block leaves; k_sort_finish then writes the identity.
//
// 16.8 M pairs: 100 to 103 us a pass (2.6 TB/s of the 16 bytes a pair moves), from
// 210 us for the count, the three scans and the scatter that it replaces.
// Bound by latency at two blocks an SM: barriers first among the waits, issue in
// 42 % of the cycles (the ballots are a third of 98 warp instructions per 32
// pairs), shared memory in 38 %.  __match_any_sync in their place
// took 57 cycles a step on its one unit per SM (155 us).  Tiles of 4096, 5120,
// 8192 pairs, 256, 512 and 1024 threads: 2 to 10 % slower.
template <int SHIFT>
__global__ void __launch_bounds__(kSortThreads, kSortBlocks) k_sort_pass(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint2 s_pair[];  // the tile's pairs in order, then per warp and digit a count
    uint32_t(*wc)[256] = reinterpret_cast<uint32_t(*)[256]>(s_pair + kSortTile);
    __shared__ uint32_t s_first[256], s_warp[8], s_tile, s_stop;
    const PassPlan plan = a.st->plan[a.pass];
    if (!plan.active) return;
    const uint32_t tiles = (uint32_t)(((uint64_t)a.n + kSortTile - 1) / kSortTile);
    for (;;) {
        if (threadIdx.x == 0) {
            s_tile = atomicAdd(&a.st->tile[a.pass], 1u);
            s_stop = load_look(&a.st->failed);
        }
        for (uint32_t k = threadIdx.x; k < kSortWarps * 256; k += kSortThreads) (&wc[0][0])[k] = 0;
        __syncthreads();
        const uint32_t tile = s_tile;
        // no tile left, or an earlier pass (or an earlier tile of this one) failed
        if (tile >= tiles || s_stop) return;
        if (threadIdx.x < 256) a.look[plan.look ^ 1u][(size_t)tile * 256 + threadIdx.x] = 0;  // for the next pass
        const uint32_t rows = (uint32_t)min((uint64_t)kSortTile, (uint64_t)a.n - (uint64_t)tile * kSortTile);
        __syncthreads();  // s_tile and s_stop have been read
        const bool ok = rows == (uint32_t)kSortTile
                            ? pass_tile<true, SHIFT>(a, plan, tile, rows, s_pair, wc, s_first, s_warp, &s_stop)
                            : pass_tile<false, SHIFT>(a, plan, tile, rows, s_pair, wc, s_first, s_warp, &s_stop);
        if (!ok) {
            if (threadIdx.x == 0) atomicAdd(&g_sort_errors, 1ull);
            return;
        }
        __syncthreads();  // the tile has left shared memory
    }
}

// Whether row x comes before row y: by the keys in order, then by row id.
__device__ __forceinline__ bool comes_before(const SortKeys &K, uint32_t x, uint32_t y)
{
    for (int k = 0; k < K.n; k++) {
        const uint64_t u = key_value(K, k, x), v = key_value(K, k, y);
        if (u != v) return u < v;
    }
    return x < y;
}

// After the head's passes: orders each run of rows that share their head (one
// thread per run, insertion).  A run longer than kTieRows sends the sort to
// all digits instead.  Streams the sorted heads once: 16.8 M rows 35 us with
// eight rows of a thread under way, 42 with one.
__global__ void __launch_bounds__(256) k_sort_ties(const __grid_constant__ SortKeys K, uint32_t n, SortState *st,
                                                    const uint32_t *word_a, const uint32_t *word_b, uint32_t *perm)
{
    if (!st->head_ran || st->head_exact || st->failed) return;
    const uint32_t *word = (st->head_ran & 1u) ? word_b : word_a;
    constexpr int kItems = 8;  // rows whose words a thread waits for at once
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i0 + 1 < n; i0 += kItems * stride) {
        uint32_t starts = 0;
#pragma unroll
        for (int j = 0; j < kItems; j++) {
            const uint64_t i = i0 + j * stride;
            const bool in = i + 1 < n;
            const uint32_t w = in ? word[i] : 0, next = in ? word[i + 1] : 0, last = in && i ? word[i - 1] : ~w;
            if (in && next == w && last != w) starts |= 1u << j;
        }
        for (; starts; starts &= starts - 1) {
            const uint64_t i = i0 + (uint64_t)(__ffs((int)starts) - 1) * stride;
            const uint32_t w = word[i];
            uint32_t len = 2;
            while (len <= kTieRows && i + len < n && word[i + len] == w) len++;
            if (len > kTieRows) {
                st->by_head = 0;
                continue;
            }
            for (uint32_t q = 1; q < len; q++) {
                const uint32_t x = perm[i + q];
                uint32_t at = q;
                for (; at > 0 && comes_before(K, x, perm[i + at - 1]); at--) perm[i + at] = perm[i + at - 1];
                perm[i + at] = x;
            }
        }
    }
}

// No active pass (all rows equal) or a failed one: the identity.
__global__ void k_sort_finish(const SortState *st, uint32_t *perm, uint32_t n)
{
    if (st->ran && !st->failed) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        perm[i] = (uint32_t)i;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct Scratch {
    SortState *st;
    uint32_t *look[2], *perm_b, *word[2];
};

size_t scratch_layout(uint64_t n, char *base, Scratch *s)
{
    const uint64_t rows = std::max<uint64_t>(n, 1);
    const uint64_t tiles = (rows + kSortTile - 1) / kSortTile;
    size_t off = 0;
    auto take = [&](uint64_t bytes) {
        char *p = base ? base + off : nullptr;
        off += align256(bytes);
        return p;
    };
    Scratch t;
    t.st = reinterpret_cast<SortState *>(take(sizeof(SortState)));
    for (int q = 0; q < 2; q++) t.look[q] = reinterpret_cast<uint32_t *>(take(tiles * 256 * 4));
    t.perm_b = reinterpret_cast<uint32_t *>(take(rows * 4));
    for (int q = 0; q < 2; q++) t.word[q] = reinterpret_cast<uint32_t *>(take(rows * 4));
    if (s) *s = t;
    return off;
}

}  // namespace

extern "C" {

size_t sdb_sort_scratch_bytes(uint64_t n) { return n <= kSmallSort ? 256 : scratch_layout(n, nullptr, nullptr); }

int sdb_sort_rows(const void *const *keys, const int *key_types, const int *descending, int nkeys, uint64_t n,
                  uint32_t *perm, void *scratch, size_t scratch_bytes, sdb_stream_t stream)
{
    return sdb_sort_rows_polls(keys, key_types, descending, nkeys, n, perm, scratch, scratch_bytes, kLookLimit, stream);
}

int sdb_sort_rows_polls(const void *const *keys, const int *key_types, const int *descending, int nkeys, uint64_t n,
                        uint32_t *perm, void *scratch, size_t scratch_bytes, uint32_t polls, sdb_stream_t stream)
{
    if (nkeys < 1 || nkeys > kMaxKeys || !keys || !key_types || !descending)
        return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_rows: 1..16 keys with types and directions");
    if (n > (1ull << 31)) return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_rows: at most 2^31 rows");
    if (n == 0) return SDB_OK;
    if (!perm || !sdb::aligned(perm, 4)) return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_rows: perm NULL or misaligned");
    const size_t need = sdb_sort_scratch_bytes(n);
    if (!scratch || scratch_bytes < need || !sdb::aligned(scratch, 256))
        return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_rows: scratch of %zu bytes (256-byte aligned) needed", need);
    SortKeys K{};
    K.n = nkeys;
    int words = 0;
    for (int k = 0; k < nkeys; k++) {
        if (key_types[k] != 0 && key_types[k] != 1)
            return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_rows: key type %d (0 int32, 1 uint64)", key_types[k]);
        if (!keys[k] || !sdb::aligned(keys[k], key_types[k] ? 8 : 4))
            return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_rows: key %d NULL or misaligned", k);
        K.col[k] = keys[k];
        K.wide[k] = key_types[k] ? 1 : 0;
        K.desc[k] = descending[k] ? 1 : 0;
        words += key_types[k] ? 2 : 1;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t n32 = (uint32_t)n;
    if (n <= kSmallSort) {
        constexpr uint32_t per_block = kSmallThreads / 32 * kSmallRows;
        k_sort_small<false><<<(n32 + per_block - 1) / per_block, kSmallThreads, 0, s>>>(K, n32, perm, SmallGather{});
        return sdb_check_launch("sdb_sort_rows");
    }
    Scratch sc;
    scratch_layout(n, static_cast<char *>(scratch), &sc);
    // a block takes tiles until none is left
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + kSortTile - 1) / kSortTile, (uint64_t)sdb::device_sms() * kSortBlocks);
    // the state and the first look-back words (adjacent) start at zero
    if (cudaMemsetAsync(sc.st, 0, reinterpret_cast<char *>(sc.look[1]) - reinterpret_cast<char *>(sc.st), s) != cudaSuccess)
        return sdb_set_error(SDB_ERR_CUDA, "sdb_sort_rows: memset failed");
    constexpr int kPassSmem = (2 * kSortTile + kSortWarps * 256) * 4;
    static sdb::SmemLimit smem_limit;
    if (!smem_limit.allow(kPassSmem, k_sort_pass<0>, k_sort_pass<8>, k_sort_pass<16>, k_sort_pass<24>))
        return sdb_set_error(SDB_ERR_CUDA, "sdb_sort_rows: shared memory size refused");
    const int passes = words * 4;
    const unsigned hist_blocks = sdb::grid_for((n + 3) / 4, kHistThreads, 8);
    PassArgs a{};
    a.n = n32;
    a.polls = polls;
    a.st = sc.st;
    for (int q = 0; q < 2; q++) {
        a.look[q] = sc.look[q];
        a.word[q] = sc.word[q];
    }
    a.perm[0] = perm;
    a.perm[1] = sc.perm_b;
    auto word_passes = [&](int k, int hi) {
        a.col = keys[k];
        a.wide = K.wide[k];
        a.desc = K.desc[k];
        a.hi = hi;
        k_sort_pass<0><<<blocks, kSortThreads, kPassSmem, s>>>(a);
        a.pass++;
        k_sort_pass<8><<<blocks, kSortThreads, kPassSmem, s>>>(a);
        a.pass++;
        k_sort_pass<16><<<blocks, kSortThreads, kPassSmem, s>>>(a);
        a.pass++;
        k_sort_pass<24><<<blocks, kSortThreads, kPassSmem, s>>>(a);
        a.pass++;
        sdb_count_launches(4);
    };
    for (int k = 0; k < nkeys; k++) k_sort_range<<<hist_blocks, kHistThreads, 0, s>>>(K, k, n32, sc.st);
    k_sort_head<<<hist_blocks, kHistThreads, 0, s>>>(K, n32, sc.st, sc.word[0]);
    k_sort_plan<<<1, 256, 0, s>>>(sc.st, 1, kHeadPasses, n32);
    a.pass = kFullPasses;
    word_passes(0, 0);
    k_sort_ties<<<sdb::grid_for(n, 256, 8), 256, 0, s>>>(K, n32, sc.st, sc.word[0], sc.word[1], perm);
    // all digits of all words, unless the rows are in order already
    k_sort_hist<<<dim3(hist_blocks, (unsigned)nkeys), kHistThreads, 0, s>>>(K, n32, sc.st);
    k_sort_plan<<<1, 256, 0, s>>>(sc.st, 0, passes, n32);
    sdb_count_launches((unsigned)nkeys + 5);
    a.pass = 0;
    for (int k = nkeys - 1; k >= 0; k--)
        for (int hi = 0; hi <= K.wide[k]; hi++) word_passes(k, hi);
    k_sort_finish<<<sdb::grid_for(n, 256, 8), 256, 0, s>>>(sc.st, perm, n32);
    return sdb_check_launch("sdb_sort_rows");
}

}  // extern "C"

// The device word that is not zero when a wait of the sort of n rows on this
// scratch ran out (its order is then 0..n-1); NULL: no such sort waits.
const uint32_t *sdb_sort_failed(uint64_t n, void *scratch)
{
    if (n <= kSmallSort) return nullptr;
    Scratch sc;
    scratch_layout(n, static_cast<char *>(scratch), &sc);
    return &sc.st->failed;
}

// The rows of a result (*count of them, on the device, at most cap to be
// ordered; cap <= 4096, up to 8 columns) written to dst in the order of the
// keys, *count_out = *count: sdb_sort_rows and a gather per column in one
// launch that needs no count on the host.  With more than cap rows only the
// count is written.
int sdb_sort_gather_small(const void *const *keys, const int *key_types, const int *descending, int nkeys,
                          const uint32_t *count, uint64_t cap, int ncols, const void *const *src, const int *wide,
                          void *const *dst, uint32_t *count_out, cudaStream_t s)
{
    if (nkeys < 1 || nkeys > kMaxKeys || cap > kSmallSort || ncols < 0 || ncols > 8)
        return sdb_set_error(SDB_ERR_INVALID, "sdb_sort_gather_small: limits exceeded");
    SortKeys K{};
    K.n = nkeys;
    for (int k = 0; k < nkeys; k++) {
        K.col[k] = keys[k];
        K.wide[k] = key_types[k] ? 1 : 0;
        K.desc[k] = descending[k] ? 1 : 0;
    }
    SmallGather G{};
    G.count = count;
    G.cap = (uint32_t)cap;
    G.count_out = count_out;
    G.ncols = ncols;
    for (int c = 0; c < ncols; c++) {
        G.src[c] = src[c];
        G.dst[c] = dst[c];
        G.wide[c] = wide[c] ? 1 : 0;
    }
    constexpr uint32_t per_block = kSmallThreads / 32 * kSmallRows;
    const uint32_t blocks = std::max<uint32_t>(1, ((uint32_t)cap + per_block - 1) / per_block);
    k_sort_small<true><<<blocks, kSmallThreads, 0, s>>>(K, 0, nullptr, G);
    return sdb_check_launch("sdb_sort_rows");
}
