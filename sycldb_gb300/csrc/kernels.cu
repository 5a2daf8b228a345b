// Operator kernels K1-K16 of the C ABI (include/sycldb_gpu.h) for sm_103a.
//
// Every kernel streams HBM: int32 columns are read with 128-bit loads
// (two int4 per 8-row group) and bool flags 8 at a time (one 64-bit word),
// grids are a multiple of the SM count and loop grid-stride.  Pointers that
// are not 16-byte (columns) / 8-byte (flags) aligned take the scalar
// instantiation, which computes the same values.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <initializer_list>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"
#include "ssbgen.cuh"

namespace {

__device__ unsigned long long g_errors;  // out-of-range slots skipped

unsigned long long read_errors(cudaStream_t s)
{
    unsigned long long v = 0, zero = 0;
    cudaMemcpyFromSymbolAsync(&v, g_errors, sizeof v, 0, cudaMemcpyDeviceToHost, s);
    cudaMemcpyToSymbolAsync(g_errors, &zero, sizeof zero, 0, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
    return v;
}
const int g_reader_registered = (sdb_errors_add_reader(&read_errors), 0);

constexpr int kThreads = 256;
constexpr int kMaxBlock = 512;  // largest block an operator kernel is tuned to

// Launch shape of an operator kernel: threads per block and the resident
// blocks per SM its grid-stride grid is sized for.  Tuned per (operator,
// log2 rows) by the autotuner (sdb_op_tune_set); unset entries take the
// defaults (256 threads; 8 blocks per SM for the map kernels, 4 for the
// reductions).
struct LaunchShape {
    int block, per_sm;
};
std::atomic<int32_t> g_op_tune[SDB_OPK_COUNT][40];  // block << 8 | per_sm; 0: default

int op_bucket(uint64_t n)
{
    int b = 0;
    while (b < 39 && (1ull << (b + 1)) <= n) b++;
    return b;
}

LaunchShape op_shape(int opk, uint64_t rows, int default_per_sm)
{
    const int32_t e = g_op_tune[opk][op_bucket(rows)].load(std::memory_order_relaxed);
    if (e <= 0) return {kThreads, default_per_sm};
    return {e >> 8, e & 0xff};
}

// Grid of `work` items for a launch shape (grid-stride kernels).
unsigned grid_of(uint64_t work, const LaunchShape &sh) { return sdb::grid_for(work, sh.block, sh.per_sm); }

// ---------------------------------------------------------------- vector io
__device__ __forceinline__ void ld8(const int32_t *p, uint64_t r0, int32_t (&v)[8])
{
    const int4 *q = reinterpret_cast<const int4 *>(p + r0);
    int4 a = __ldcs(q), b = __ldcs(q + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

__device__ __forceinline__ void st8(int32_t *p, uint64_t r0, const int32_t (&v)[8])
{
    int4 *q = reinterpret_cast<int4 *>(p + r0);
    q[0] = make_int4(v[0], v[1], v[2], v[3]);
    q[1] = make_int4(v[4], v[5], v[6], v[7]);
}

__device__ __forceinline__ uint32_t nz_bits4(uint32_t w)
{
    uint32_t x = __vcmpne4(w, 0u);
    return ((x >> 7) & 1u) | ((x >> 14) & 2u) | ((x >> 21) & 4u) | ((x >> 28) & 8u);
}

__device__ __forceinline__ uint32_t ldf8(const uint8_t *p, uint64_t r0)
{
    uint2 w = __ldcs(reinterpret_cast<const uint2 *>(p + r0));
    return nz_bits4(w.x) | (nz_bits4(w.y) << 4);
}

__device__ __forceinline__ uint32_t bits_to_bytes4(uint32_t m)
{
    return (m & 1u) | ((m & 2u) << 7) | ((m & 4u) << 14) | ((m & 8u) << 21);
}

__device__ __forceinline__ void stf8(uint8_t *p, uint64_t r0, uint32_t m)
{
    uint2 w;
    w.x = bits_to_bytes4(m & 0xFu);
    w.y = bits_to_bytes4((m >> 4) & 0xFu);
    *reinterpret_cast<uint2 *>(p + r0) = w;
}

// Grid-stride driver: Op provides group(r0) for 8 rows (vector path) and
// row(r) for one row.  VEC=false walks rows one at a time.
template <bool VEC, class Op>
__global__ void __launch_bounds__(kMaxBlock) k_map(uint64_t n, Op op)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    if (VEC) {
        const uint64_t groups = n >> 3;
        for (uint64_t g = tid; g < groups; g += stride) op.group(g << 3);
        for (uint64_t r = (groups << 3) + tid; r < n; r += stride) op.row(r);
    } else {
        for (uint64_t r = tid; r < n; r += stride) op.row(r);
    }
}

template <class Op>
int launch_map(uint64_t n, bool vec, const Op &op, cudaStream_t s, const char *what, int opk)
{
    if (n == 0) return SDB_OK;
    const LaunchShape sh = op_shape(opk, n, 8);
    if (vec)
        k_map<true, Op><<<grid_of((n + 7) / 8, sh), sh.block, 0, s>>>(n, op);
    else
        k_map<false, Op><<<grid_of(n, sh), sh.block, 0, s>>>(n, op);
    return sdb_check_launch(what);
}

// ---------------------------------------------------------------- K1, K5
struct FillU8 {
    uint8_t *f; uint8_t v;
    __device__ void group(uint64_t r0) const
    {
        uint32_t w = 0x01010101u * v;
        *reinterpret_cast<uint2 *>(f + r0) = make_uint2(w, w);
    }
    __device__ void row(uint64_t r) const { f[r] = v; }
};

struct FillI32 {
    int32_t *d; int32_t v;
    __device__ void group(uint64_t r0) const
    {
        int32_t x[8] = {v, v, v, v, v, v, v, v};
        st8(d, r0, x);
    }
    __device__ void row(uint64_t r) const { d[r] = v; }
};

// ---------------------------------------------------------------- K2, K3, K4
struct SelectLit {
    const int32_t *col; int32_t v; int cmp, logic; const uint8_t *in; uint8_t *out;
    __device__ void group(uint64_t r0) const
    {
        int32_t c[8];
        ld8(col, r0, c);
        uint32_t fin = ldf8(in, r0), m = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) m |= (uint32_t)sdb::compare(cmp, c[j], v) << j;
        uint32_t lo = sdb::logical4(logic, fin & 0xF, m & 0xF), hi = sdb::logical4(logic, fin >> 4, m >> 4);
        stf8(out, r0, lo | (hi << 4));
    }
    __device__ void row(uint64_t r) const { out[r] = sdb::logical(logic, in[r] != 0, sdb::compare(cmp, col[r], v)); }
};

struct SelectCols {
    const int32_t *a, *b; int cmp, logic; const uint8_t *in; uint8_t *out;
    __device__ void group(uint64_t r0) const
    {
        int32_t x[8], y[8];
        ld8(a, r0, x);
        ld8(b, r0, y);
        uint32_t fin = ldf8(in, r0), m = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) m |= (uint32_t)sdb::compare(cmp, x[j], y[j]) << j;
        uint32_t lo = sdb::logical4(logic, fin & 0xF, m & 0xF), hi = sdb::logical4(logic, fin >> 4, m >> 4);
        stf8(out, r0, lo | (hi << 4));
    }
    __device__ void row(uint64_t r) const { out[r] = sdb::logical(logic, in[r] != 0, sdb::compare(cmp, a[r], b[r])); }
};

struct Logical {
    int logic; const uint8_t *in, *local; uint8_t *out;
    __device__ void group(uint64_t r0) const
    {
        uint32_t a = ldf8(in, r0), b = ldf8(local, r0);
        uint32_t lo = sdb::logical4(logic, a & 0xF, b & 0xF), hi = sdb::logical4(logic, a >> 4, b >> 4);
        stf8(out, r0, lo | (hi << 4));
    }
    __device__ void row(uint64_t r) const { out[r] = sdb::logical(logic, in[r] != 0, local[r] != 0); }
};

// ---------------------------------------------------------------- K6
// mode 0: col op col, 1: lit op col, 2: col op lit
struct Binop {
    int32_t *res; const int32_t *a, *b; int32_t la, lb; int op, mode; const uint8_t *flags;
    __device__ int32_t A(uint64_t r) const { return mode == 1 ? la : a[r]; }
    __device__ int32_t B(uint64_t r) const { return mode == 2 ? lb : b[r]; }
    __device__ void group(uint64_t r0) const
    {
        uint32_t f = ldf8(flags, r0);
        if (f == 0) return;
        int32_t x[8], y[8];
        if (mode == 1) { for (int j = 0; j < 8; j++) x[j] = la; } else ld8(a, r0, x);
        if (mode == 2) { for (int j = 0; j < 8; j++) y[j] = lb; } else ld8(b, r0, y);
        if (f == 0xFFu) {
            int32_t z[8];
#pragma unroll
            for (int j = 0; j < 8; j++) z[j] = sdb::binop(x[j], y[j], op);
            st8(res, r0, z);
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (f & (1u << j)) res[r0 + j] = sdb::binop(x[j], y[j], op);
        }
    }
    __device__ void row(uint64_t r) const
    {
        if (flags[r]) res[r] = sdb::binop(A(r), B(r), op);
    }
};

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v)
{
    __shared__ uint64_t part[kMaxBlock / 32];
    v = warp_sum_u64(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) part[wid] = v;
    __syncthreads();
    uint64_t t = 0;
    if (wid == 0) {
        t = lane < (int)(blockDim.x >> 5) ? part[lane] : 0;
        t = warp_sum_u64(t);
    }
    __syncthreads();
    return t;  // valid in thread 0
}

// K7: one 64-bit atomic per block.
template <bool VEC>
__global__ void __launch_bounds__(kMaxBlock) k_sum(const int32_t *col, const uint8_t *flags, uint64_t n, uint64_t *acc)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t s = 0;
    uint64_t start = 0;
    if (VEC) {
        const uint64_t groups = n >> 3;
        for (uint64_t g = tid; g < groups; g += stride) {
            uint32_t f = ldf8(flags, g << 3);
            if (f == 0) continue;
            int32_t c[8];
            ld8(col, g << 3, c);
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (f & (1u << j)) s += sdb::widen(c[j]);
        }
        start = groups << 3;
    }
    for (uint64_t r = start + tid; r < n; r += stride)
        if (flags[r]) s += sdb::widen(col[r]);
    s = block_sum_u64(s);
    if (threadIdx.x == 0 && s != 0) atomicAdd(reinterpret_cast<unsigned long long *>(acc), (unsigned long long)s);
}

// K16
template <bool VEC>
__global__ void __launch_bounds__(kMaxBlock) k_count(const uint8_t *flags, uint64_t n, uint64_t *out)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t s = 0, start = 0;
    if (VEC) {
        const uint64_t groups = n >> 3;
        for (uint64_t g = tid; g < groups; g += stride) s += __popc(ldf8(flags, g << 3));
        start = groups << 3;
    }
    for (uint64_t r = start + tid; r < n; r += stride) s += flags[r] != 0;
    s = block_sum_u64(s);
    if (threadIdx.x == 0 && s != 0) atomicAdd(reinterpret_cast<unsigned long long *>(out), (unsigned long long)s);
}

// min/max at load
__global__ void k_minmax_init(int32_t *mm)
{
    mm[0] = INT32_MAX;
    mm[1] = INT32_MIN;
}

template <bool VEC>
__global__ void __launch_bounds__(kMaxBlock) k_minmax(const int32_t *col, uint64_t n, int32_t *mm)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    int32_t lo = INT32_MAX, hi = INT32_MIN;
    uint64_t start = 0;
    if (VEC) {
        const uint64_t groups = n >> 3;
        for (uint64_t g = tid; g < groups; g += stride) {
            int32_t c[8];
            ld8(col, g << 3, c);
#pragma unroll
            for (int j = 0; j < 8; j++) { lo = min(lo, c[j]); hi = max(hi, c[j]); }
        }
        start = groups << 3;
    }
    for (uint64_t r = start + tid; r < n; r += stride) { lo = min(lo, col[r]); hi = max(hi, col[r]); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&mm[0], lo);
        atomicMax(&mm[1], hi);
    }
}

// ---------------------------------------------------------------- K8, K9
struct GroupArgs {
    const int32_t *keys[8];
    int32_t mins[8];
    uint32_t mults[8];
    int g;
    const int32_t *val;
    const uint8_t *flags;
    uint64_t n, P;
    int32_t *out_keys[8];
    uint64_t *out_sum;
    uint32_t *occ;
};

__device__ __forceinline__ int64_t row_slot(const GroupArgs &a, uint64_t r)
{
    uint32_t h = 0;
#pragma unroll
    for (int j = 0; j < 8; j++)
        if (j < a.g) h += ((uint32_t)a.keys[j][r] - (uint32_t)a.mins[j]) * a.mults[j];
    return sdb::group_slot(h, a.P);
}

__device__ __forceinline__ void claim_keys(const GroupArgs &a, int64_t h, uint64_t r)
{
    if (atomicExch(&a.occ[h], 1u) == 0u)
        for (int j = 0; j < a.g; j++) a.out_keys[j][h] = a.keys[j][r];
}

// One flagged row's slot update (K8): the first writer of a slot stores its
// keys, the value goes into the slot's sum.
//
// SMEM: the sums are private to the block, in shared memory.  A block's first touch of a
// slot also runs the global first-writer exchange; sums flush once per touched
// slot.  A slot's 64-bit sum is a low and a high word (s_lo[h], s_lo[P + h])
// added with 32-bit atomics, the low word's carry taken from the value its add
// returns: 64-bit shared atomics are compare-and-swap loops (28 cycles of an SM
// per warp over 280 slots, 450 over two; 9 and 19 this way).
template <bool SMEM>
__device__ __forceinline__ void group_row(const GroupArgs &a, uint64_t r, uint32_t *s_lo, uint32_t *s_occ)
{
    const int32_t v = a.val[r];  // on its way with the keys
    const int64_t h = row_slot(a, r);
    if (h < 0 || (uint64_t)h >= a.P) {
        atomicAdd(&g_errors, 1ull);
        return;
    }
    if (SMEM) {
        if (s_occ[h] == 0u && atomicExch(&s_occ[h], 1u) == 0u) claim_keys(a, h, r);
        const uint32_t old = atomicAdd(&s_lo[h], (uint32_t)v);
        const uint32_t hi = (uint32_t)(old + (uint32_t)v < old) + (uint32_t)(v >> 31);
        if (hi) atomicAdd(&s_lo[a.P + h], hi);
    } else {
        if (a.occ[h] == 0u) claim_keys(a, h, r);
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.out_sum[h]), (unsigned long long)sdb::widen(v));
    }
}

// Clears a block's private table / adds it to the global sums.
template <int THREADS>
__device__ __forceinline__ void group_reset(const GroupArgs &a, uint32_t *s_lo)
{
    for (uint64_t i = threadIdx.x; i < 3 * a.P; i += THREADS) s_lo[i] = 0;
    __syncthreads();
}

template <int THREADS>
__device__ __forceinline__ void group_flush(const GroupArgs &a, const uint32_t *s_lo, const uint32_t *s_occ)
{
    __syncthreads();
    for (uint64_t i = threadIdx.x; i < a.P; i += THREADS)
        if (s_occ[i])
            atomicAdd(reinterpret_cast<unsigned long long *>(&a.out_sum[i]),
                      (unsigned long long)s_lo[i] | ((unsigned long long)s_lo[a.P + i] << 32));
}

// Flags of the lane's 16 rows r0 .. r0 + 15 as a mask: one 16-byte load
// (already made: q) where VEC and all 16 exist.
template <bool VEC>
__device__ __forceinline__ uint32_t group_mask(const GroupArgs &a, uint64_t r0, const uint4 &q)
{
    if (VEC && r0 + 16 <= a.n) return nz_bits4(q.x) | (nz_bits4(q.y) << 4) | (nz_bits4(q.z) << 8) | (nz_bits4(q.w) << 12);
    uint32_t m = 0;
    for (int b = 0; b < 16 && r0 + b < a.n; b++) m |= (uint32_t)(a.flags[r0 + b] != 0) << b;
    return m;
}

template <bool VEC>
__device__ __forceinline__ uint4 group_flags(const GroupArgs &a, uint64_t r0)
{
    return VEC && r0 + 16 <= a.n ? __ldcs(reinterpret_cast<const uint4 *>(a.flags + r0)) : make_uint4(0, 0, 0, 0);
}

// Queues the first row of each lane's mask (of rows r0 .. r0 + 15; `any`: the
// lanes that have one) and updates the queue's last 32 once there are as many:
// fewer than 32 before and after.
template <bool SMEM>
__device__ __forceinline__ void group_queue(const GroupArgs &a, uint32_t &m, unsigned any, uint64_t r0, uint64_t *queue,
                                            uint32_t &queued, uint32_t *s_lo, uint32_t *s_occ)
{
    const uint32_t lane = threadIdx.x & 31u;
    if (m) {
        queue[queued + __popc(any & ((1u << lane) - 1u))] = r0 + (uint32_t)__ffs(m) - 1u;
        m &= m - 1;
    }
    queued += __popc(any);
    __syncwarp();
    if (queued >= 32) {
        queued -= 32;
        const uint64_t r = queue[queued + lane];
        __syncwarp();  // read before the queue grows again
        group_row<SMEM>(a, r, s_lo, s_occ);
    }
}

// The two forms walk chunks of 512 rows a warp, 16 rows a lane.
//
// Listed: the warp lists a chunk's flagged rows in row order (a prefix sum of the
// lanes' counts) and updates them one per lane, so that the loads of a step
// fall into neighbouring sectors and the steps of a chunk do not wait for one
// another; the rows of a chunk with at most one per lane are queued over
// chunks instead.  For the slots past shared memory, where every update goes to
// the global arrays, and for inputs whose 512-thread blocks would leave SMs
// empty.
//
// Queued: every flagged row is queued over chunks and updated one per lane, 32 at a
// time, so that a warp does not wait for the key and value loads of the few
// rows of a chunk; the next chunk's flags are on their way meanwhile.  512 threads
// share a table: with P = 7000 two blocks fit an SM whatever their size.
//
// Both bound by the latency of the row loads and, where most rows are flagged,
// by the atomics.  us, listed / queued, all rows flagged and 1 in 250:
//   30 M rows, P = 100,000    297 / 398 and 17 / 16
//   30 M rows, P = 7000       476 / 252 and 25 / 19
//   400 K rows, P = 7000       21 / 25 and 6.4 / 6.5
template <bool SMEM, bool VEC>
__global__ void __launch_bounds__(kThreads) k_groupby_listed(const GroupArgs a)
{
    constexpr uint32_t kWarps = kThreads / 32;
    extern __shared__ uint32_t s_lo[];  // P low words, P high words, P occupancy words
    __shared__ uint64_t s_queue[kWarps][64];
    __shared__ uint16_t s_list[kWarps][512];
    uint32_t *s_occ = s_lo + (SMEM ? 2 * a.P : 0);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t *queue = s_queue[warp];
    uint16_t *list = s_list[warp];
    uint32_t queued = 0;  // rows in the queue (warp-uniform)
    if (SMEM) group_reset<kThreads>(a, s_lo);
    for (uint64_t c = (uint64_t)blockIdx.x * kWarps + warp; c * 512 < a.n; c += (uint64_t)gridDim.x * kWarps) {
        const uint64_t base = c * 512, r0 = base + lane * 16;
        uint32_t m = group_mask<VEC>(a, r0, group_flags<VEC>(a, r0));
        const uint32_t cnt = __popc(m);
        if (!__any_sync(0xffffffffu, cnt > 1)) {
            group_queue<SMEM>(a, m, __ballot_sync(0xffffffffu, cnt), r0, queue, queued, s_lo, s_occ);
            continue;
        }
        uint32_t pos = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, pos, o);
            if (lane >= (uint32_t)o) pos += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, pos, 31);
        pos -= cnt;
        for (; m; m &= m - 1) list[pos++] = (uint16_t)(lane * 16 + (uint32_t)__ffs(m) - 1u);
        __syncwarp();
        for (uint32_t i = lane; i < total; i += 32) group_row<SMEM>(a, base + list[i], s_lo, s_occ);
        __syncwarp();
    }
    if (lane < queued) group_row<SMEM>(a, queue[lane], s_lo, s_occ);
    if (SMEM) group_flush<kThreads>(a, s_lo, s_occ);
}

constexpr int kGroupThreads = 512;

template <bool VEC>
__global__ void __launch_bounds__(kGroupThreads) k_groupby_queued(const GroupArgs a)
{
    constexpr uint32_t kWarps = kGroupThreads / 32;
    extern __shared__ uint32_t s_lo[];  // as above
    __shared__ uint64_t s_queue[kWarps][64];
    uint32_t *s_occ = s_lo + 2 * a.P;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t *queue = s_queue[warp];
    uint32_t queued = 0;
    group_reset<kGroupThreads>(a, s_lo);
    const uint64_t wstride = (uint64_t)gridDim.x * kWarps;
    uint64_t c = (uint64_t)blockIdx.x * kWarps + warp;
    uint4 next = group_flags<VEC>(a, c * 512 + lane * 16);
    for (; c * 512 < a.n; c += wstride) {
        const uint64_t r0 = c * 512 + lane * 16;
        uint32_t m = group_mask<VEC>(a, r0, next);
        next = group_flags<VEC>(a, r0 + wstride * 512);
        while (const unsigned any = __ballot_sync(0xffffffffu, m != 0))
            group_queue<true>(a, m, any, r0, queue, queued, s_lo, s_occ);
    }
    if (lane < queued) group_row<true>(a, queue[lane], s_lo, s_occ);
    group_flush<kGroupThreads>(a, s_lo, s_occ);
}

struct OccToFlags {
    const uint32_t *occ; uint8_t *f;
    __device__ void group(uint64_t r0) const
    {
        const uint4 *q = reinterpret_cast<const uint4 *>(occ + r0);
        uint4 a = q[0], b = q[1];
        uint32_t m = (a.x != 0) | ((a.y != 0) << 1) | ((a.z != 0) << 2) | ((a.w != 0) << 3) |
                     ((b.x != 0) << 4) | ((b.y != 0) << 5) | ((b.z != 0) << 6) | ((b.w != 0) << 7);
        stf8(f, r0, m);
    }
    __device__ void row(uint64_t r) const { f[r] = occ[r] != 0; }
};

// ---------------------------------------------------------------- K10 - K13
__global__ void __launch_bounds__(kMaxBlock) k_build_keys(const int32_t *key, const uint8_t *flags, uint64_t n,
                                                         uint8_t *ht, int32_t mn, int32_t len)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        int64_t h = sdb::ht_slot(key[r], len, mn);
        if (h < 0 || h >= len) { atomicAdd(&g_errors, 1ull); continue; }
        ht[h] = flags[r] ? 1 : 0;
    }
}

__global__ void __launch_bounds__(kMaxBlock) k_build_kv(const int32_t *key, const int32_t *val, const uint8_t *flags,
                                                       uint64_t n, int32_t *ht2, int32_t mn, int32_t len)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        int64_t h = sdb::ht_slot(key[r], len, mn);
        if (h < 0 || h >= len) { atomicAdd(&g_errors, 1ull); continue; }
        if (flags[r]) {
            ht2[2 * h] = 1;
            ht2[2 * h + 1] = val[r];
        } else {
            ht2[2 * h] = 0;
        }
    }
}

struct ProbeSemi {
    const int32_t *key; const uint8_t *in; uint8_t *out; const uint8_t *ht; int32_t mn, mx;
    __device__ bool one(int32_t k, bool fin) const
    {
        return fin && k >= mn && k <= mx && __ldg(ht + ((uint32_t)k - (uint32_t)mn)) != 0;
    }
    __device__ void group(uint64_t r0) const
    {
        uint32_t f = ldf8(in, r0), m = 0;
        if (f) {
            int32_t k[8];
            ld8(key, r0, k);
#pragma unroll
            for (int j = 0; j < 8; j++) m |= (uint32_t)one(k[j], (f >> j) & 1u) << j;
        }
        stf8(out, r0, m);
    }
    __device__ void row(uint64_t r) const { out[r] = in[r] ? one(key[r], true) : 0; }
};

template <bool HT8>
struct ProbeFull {
    const int32_t *key; int32_t *val_out; const uint8_t *in; uint8_t *out; const int32_t *ht2; int32_t mn, mx;
    __device__ bool one(int32_t k, bool fin, int32_t &v) const
    {
        if (!fin || k < mn || k > mx) return false;
        const uint32_t h = (uint32_t)k - (uint32_t)mn;
        int32_t occ, val;
        if (HT8) {
            int2 e = __ldg(reinterpret_cast<const int2 *>(ht2) + h);
            occ = e.x; val = e.y;
        } else {
            occ = __ldg(ht2 + 2 * (uint64_t)h);
            val = __ldg(ht2 + 2 * (uint64_t)h + 1);
        }
        v = val;
        return occ == 1;
    }
    __device__ void group(uint64_t r0) const
    {
        uint32_t f = ldf8(in, r0), m = 0;
        if (f) {
            int32_t k[8];
            ld8(key, r0, k);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                int32_t v;
                if (one(k[j], (f >> j) & 1u, v)) {
                    val_out[r0 + j] = v;
                    m |= 1u << j;
                }
            }
        }
        stf8(out, r0, m);
    }
    __device__ void row(uint64_t r) const
    {
        int32_t v;
        if (in[r] && one(key[r], true, v)) {
            val_out[r] = v;
            out[r] = 1;
        } else {
            out[r] = 0;
        }
    }
};

// ------------------------------------------- K10 - K13 on open-addressing tables
// The same builds and probes over a table of 2^lg slots (sdb::oa_put /
// oa_find): a build row writes its key's slot as the direct-address build
// writes key - min (live: hit and value, dead: miss); `fresh` (the table is
// all zero and no other build writes it) skips dead rows, whose miss the
// empty table already reads.
__global__ void __launch_bounds__(kMaxBlock) k_build_keys_oa(const int32_t *key, const uint8_t *flags, uint64_t n,
                                                            uint32_t *ht, int lg, int32_t mn, int32_t mx, int fresh)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const bool live = flags[r] != 0;
        if (!live && fresh) continue;
        const int32_t k = key[r];
        if (k < mn || k > mx || sdb::oa_put<1>(ht, lg, sdb::oa_tag(k, mn), live) == -2) atomicAdd(&g_errors, 1ull);
    }
}

__global__ void __launch_bounds__(kMaxBlock) k_build_kv_oa(const int32_t *key, const int32_t *val, const uint8_t *flags,
                                                          uint64_t n, int32_t *ht2, int lg, int32_t mn, int32_t mx,
                                                          int fresh)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const bool live = flags[r] != 0;
        if (!live && fresh) continue;
        const int32_t k = key[r];
        if (k < mn || k > mx) {
            atomicAdd(&g_errors, 1ull);
            continue;
        }
        const int64_t h = sdb::oa_put<2>(reinterpret_cast<uint32_t *>(ht2), lg, sdb::oa_tag(k, mn), live);
        if (h == -2) atomicAdd(&g_errors, 1ull);
        else if (h >= 0 && live) ht2[2 * h + 1] = val[r];
    }
}

struct ProbeSemiOA {
    const int32_t *key; const uint8_t *in; uint8_t *out; const uint32_t *ht; int lg; int32_t mn, mx;
    __device__ bool one(int32_t k, bool fin) const
    {
        if (!fin || k < mn || k > mx) return false;
        const int64_t h = sdb::oa_find<1>(ht, lg, sdb::oa_tag(k, mn));
        return h >= 0 && (__ldg(ht + h) & 1u);
    }
    __device__ void group(uint64_t r0) const
    {
        uint32_t f = ldf8(in, r0), m = 0;
        if (f) {
            int32_t k[8];
            ld8(key, r0, k);
#pragma unroll
            for (int j = 0; j < 8; j++) m |= (uint32_t)one(k[j], (f >> j) & 1u) << j;
        }
        stf8(out, r0, m);
    }
    __device__ void row(uint64_t r) const { out[r] = in[r] ? one(key[r], true) : 0; }
};

struct ProbeFullOA {
    const int32_t *key; int32_t *val_out; const uint8_t *in; uint8_t *out; const int32_t *ht2; int lg; int32_t mn, mx;
    __device__ bool one(int32_t k, bool fin, int32_t &v) const
    {
        if (!fin || k < mn || k > mx) return false;
        const int64_t h = sdb::oa_find<2>(reinterpret_cast<const uint32_t *>(ht2), lg, sdb::oa_tag(k, mn));
        if (h < 0) return false;
        const int2 e = __ldg(reinterpret_cast<const int2 *>(ht2) + h);
        v = e.y;
        return (e.x & 1) != 0;
    }
    __device__ void group(uint64_t r0) const
    {
        uint32_t f = ldf8(in, r0), m = 0;
        if (f) {
            int32_t k[8];
            ld8(key, r0, k);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                int32_t v;
                if (one(k[j], (f >> j) & 1u, v)) {
                    val_out[r0 + j] = v;
                    m |= 1u << j;
                }
            }
        }
        stf8(out, r0, m);
    }
    __device__ void row(uint64_t r) const
    {
        int32_t v;
        if (in[r] && one(key[r], true, v)) {
            val_out[r] = v;
            out[r] = 1;
        } else {
            out[r] = 0;
        }
    }
};

// ---------------------------------------------------------------- K14, K15
// Ordered compaction: the flagged rows of a segment, in row order, as row ids
// and / or gathered columns.  Two launches: the tiles' counts, then every tile
// adds up the counts of the tiles before it (at most 4096 words, from L2) and
// writes its rows.  Streams the flags twice; the second time they come from
// L2 up to its size.  The row list in shared memory makes the gathers and the
// stores consecutive.  30 M flags, 0.36 % set, two int32 columns: 32 us; with a
// one-block scan of the counts between the two and a gather launch per
// column on top it was 65.
constexpr int kCompactRowsPerThread = 16;
constexpr int kCompactChunk = kThreads * kCompactRowsPerThread;  // rows per count that callers' scratch is sized for
constexpr uint32_t kCompactRows = 4 * kCompactChunk;              // most rows a block lists at a time
constexpr uint32_t kCompactTiles = 4096;                          // most tiles of a launch
constexpr int kCompactCols = 8;                                   // columns gathered by one launch

struct Compact {
    const void *flags;  // uint8 flags, or uint32 occupancy words (flag = word != 0)
    uint64_t n;
    uint32_t steps;     // 16-row steps of a thread per list: 4, or 1 (a quarter of kCompactRows)
    uint32_t subs;      // a tile is `subs` lists
    uint32_t *counts;   // per tile
    int32_t *ids;       // NULL: not wanted
    uint32_t *count;
    int32_t ncols;
    const void *src[kCompactCols];
    void *dst[kCompactCols];
    int32_t wide[kCompactCols];  // 1: uint64 column
};

// Flags of rows r0 .. r0 + 15 as a mask (r0 a multiple of 16, flags 16-byte aligned).
template <typename F>
__device__ __forceinline__ uint32_t mask16(const F *flags, uint64_t r0, uint64_t n)
{
    uint32_t m = 0;
    if (r0 + 16 <= n) {
        const uint4 *q = reinterpret_cast<const uint4 *>(flags + r0);
        if (sizeof(F) == 1) {
            const uint4 w = q[0];
            return nz_bits4(w.x) | (nz_bits4(w.y) << 4) | (nz_bits4(w.z) << 8) | (nz_bits4(w.w) << 12);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint4 w = q[j];
            m |= ((w.x != 0) | ((w.y != 0) << 1) | ((w.z != 0) << 2) | ((w.w != 0) << 3)) << (4 * j);
        }
        return m;
    }
    for (uint64_t r = r0; r < n; r++) m |= (uint32_t)(flags[r] != 0) << (r - r0);
    return m;
}

// Exclusive block scan of one value per thread; returns the block total in *total.
template <int THREADS>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t warp_tot[THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    uint32_t base = 0, all = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; w++) {
        const uint32_t t = warp_tot[w];
        base += w < wid ? t : 0;
        all += t;
    }
    *total = all;
    __syncthreads();
    return base + x - v;
}

// Writes the rows list[0 .. total) (offsets from r0) at positions pos ..
template <int THREADS>
__device__ __forceinline__ void put_rows(const Compact &a, const uint16_t *list, uint32_t total, uint64_t r0, uint32_t pos)
{
    for (uint32_t i = threadIdx.x; i < total; i += THREADS) {
        const uint64_t r = r0 + list[i];
        const uint32_t at = pos + i;
        if (a.ids) a.ids[at] = (int32_t)r;
        // every column loaded before any store
        uint64_t v[kCompactCols];
#pragma unroll
        for (int c = 0; c < kCompactCols; c++)
            if (c < a.ncols)
                v[c] = a.wide[c] ? static_cast<const uint64_t *>(a.src[c])[r]
                                 : (uint64_t)(uint32_t)static_cast<const int32_t *>(a.src[c])[r];
#pragma unroll
        for (int c = 0; c < kCompactCols; c++)
            if (c < a.ncols) {
                if (a.wide[c]) static_cast<uint64_t *>(a.dst[c])[at] = v[c];
                else static_cast<int32_t *>(a.dst[c])[at] = (int32_t)(uint32_t)v[c];
            }
    }
}

template <typename F>
__global__ void __launch_bounds__(kThreads) k_compact_count(const __grid_constant__ Compact a)
{
    const uint64_t list_rows = (uint64_t)a.steps * kCompactChunk, t0 = blockIdx.x * a.subs * list_rows;
    uint32_t c = 0;
    for (uint32_t s = 0; s < a.subs; s++) {
        const uint64_t r0 = t0 + s * list_rows + threadIdx.x * 16u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint64_t r = r0 + (uint64_t)j * kCompactChunk;
            if (j < (int)a.steps && r < a.n) c += __popc(mask16(static_cast<const F *>(a.flags), r, a.n));
        }
    }
    uint32_t total;
    block_exclusive_scan<kThreads>(c, &total);
    if (threadIdx.x == 0) a.counts[blockIdx.x] = total;
}

template <typename F>
__global__ void __launch_bounds__(kThreads) k_compact_write(const __grid_constant__ Compact a)
{
    __shared__ uint16_t s_list[kCompactRows];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t list_rows = (uint64_t)a.steps * kCompactChunk, t0 = blockIdx.x * a.subs * list_rows;
    // warp w lists rows [512 steps w, 512 steps (w + 1)): steps of 16 rows per lane
    const uint32_t first = warp * 512u * a.steps + lane * 16u;
    uint32_t m[4];
    auto load = [&](uint64_t r0) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint64_t r = r0 + first + j * 512u;
            m[j] = j < (int)a.steps && r < a.n ? mask16(static_cast<const F *>(a.flags), r, a.n) : 0;
        }
    };
    load(t0);  // in flight with the counts
    uint32_t before = 0, pos;
#pragma unroll 4
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kThreads) before += a.counts[t];
    block_exclusive_scan<kThreads>(before, &pos);
    for (uint32_t s = 0; s < a.subs; s++) {
        const uint64_t r0 = t0 + s * list_rows;
        if (r0 >= a.n) break;  // block-uniform
        if (s) load(r0);
        // the steps' lane prefixes, two 16-bit counts a word (at most 512 each)
        uint32_t x = __popc(m[0]) | (__popc(m[1]) << 16), y = __popc(m[2]) | (__popc(m[3]) << 16);
        const uint32_t cx = x, cy = y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t px = __shfl_up_sync(0xffffffffu, x, o), py = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= (uint32_t)o) {
                x += px;
                y += py;
            }
        }
        const uint32_t tx = __shfl_sync(0xffffffffu, x, 31), ty = __shfl_sync(0xffffffffu, y, 31);
        const uint32_t sums[4] = {tx & 0xffffu, tx >> 16, ty & 0xffffu, ty >> 16};
        x -= cx;
        y -= cy;
        const uint32_t lanes[4] = {x & 0xffffu, x >> 16, y & 0xffffu, y >> 16};
        uint32_t total;
        uint32_t at = block_exclusive_scan<kThreads>(lane == 0 ? sums[0] + sums[1] + sums[2] + sums[3] : 0, &total);
        at = __shfl_sync(0xffffffffu, at, 0);  // lane 0's prefix is its warp's
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t q = at + lanes[j], f = m[j];
            while (f) {
                s_list[q++] = (uint16_t)(first + j * 512u + (uint32_t)__ffs(f) - 1u);
                f &= f - 1;
            }
            at += sums[j];
        }
        __syncthreads();
        put_rows<kThreads>(a, s_list, total, r0, pos);
        pos += total;
        __syncthreads();  // the list has been read
    }
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) *a.count = pos;
}

template <typename T>
__global__ void __launch_bounds__(kMaxBlock) k_gather(const T *src, const int32_t *ids, const uint32_t *count, T *dst,
                                                     uint64_t cap)
{
    const uint64_t c = min((uint64_t)*count, cap);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < c; i += stride) dst[i] = src[ids[i]];
}

// The same for a small segment (a group-by result) in one launch: every block
// counts the flags before its 2048 rows itself.  4375 slots, four columns:
// 6.3 us, 8.5 in one block of 1024 threads with a thread's rows side by side.
constexpr uint32_t kSmallCompactMax = 65536;
constexpr int kSmallCompactThreads = 512;

template <typename F, bool VEC>
__global__ void __launch_bounds__(kSmallCompactThreads) k_compact_gather_small(const __grid_constant__ Compact a)
{
    __shared__ uint16_t s_list[4 * kSmallCompactThreads];
    const F *flags = static_cast<const F *>(a.flags);
    const uint32_t n = (uint32_t)a.n, r0 = blockIdx.x * 4u * kSmallCompactThreads;
    // flags of rows r .. r + 3 as a mask
    auto mask4 = [&](uint32_t r) -> uint32_t {
        if (VEC && r + 4 <= n) {
            if (sizeof(F) == 1) return nz_bits4(*reinterpret_cast<const uint32_t *>(flags + r));
            const uint4 w = *reinterpret_cast<const uint4 *>(flags + r);
            return (w.x != 0) | ((w.y != 0) << 1) | ((w.z != 0) << 2) | ((w.w != 0) << 3);
        }
        uint32_t m = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++)
            if (r + j < n) m |= (uint32_t)(flags[r + j] != 0) << j;
        return m;
    };
    uint32_t before = 0;
    uint32_t m = mask4(r0 + threadIdx.x * 4u);
#pragma unroll 8
    for (uint32_t b = 0; b < blockIdx.x; b++) before += __popc(mask4((b * kSmallCompactThreads + threadIdx.x) * 4u));
    uint32_t pos, total;
    block_exclusive_scan<kSmallCompactThreads>(before, &pos);
    uint32_t at = block_exclusive_scan<kSmallCompactThreads>(__popc(m), &total);
    while (m) {
        s_list[at++] = (uint16_t)(threadIdx.x * 4u + (uint32_t)__ffs(m) - 1u);
        m &= m - 1;
    }
    __syncthreads();
    put_rows<kSmallCompactThreads>(a, s_list, total, r0, pos);
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) *a.count = pos + total;
}

// ---------------------------------------------------------------- data gen
__global__ void __launch_bounds__(kThreads) k_gen_uniform(int32_t *dst, uint64_t n, uint64_t row0, uint64_t key,
                                                          int32_t lo, int32_t hi)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = sdb::uniform_from_key(key, row0 + i, lo, hi);
}

__global__ void __launch_bounds__(kThreads) k_gen_dates(int32_t *dst, uint64_t n, uint64_t row0, uint64_t key,
                                                        int32_t ndays)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = sdb::datekey_of_day(sdb::uniform_from_key(key, row0 + i, 0, ndays - 1));
}

template <class F>
void parallel_rows(uint64_t n, F f)
{
    unsigned nt = std::thread::hardware_concurrency();
    if (nt == 0) nt = 1;
    if (n < (1u << 16)) nt = 1;
    std::vector<std::thread> th;
    uint64_t per = (n + nt - 1) / nt;
    for (unsigned t = 0; t < nt; t++) {
        uint64_t a = t * per, b = std::min<uint64_t>(n, a + per);
        if (a >= b) break;
        th.emplace_back([=] { for (uint64_t i = a; i < b; i++) f(i); });
    }
    for (auto &x : th) x.join();
}

bool flags_ok(const uint8_t *p) { return sdb::aligned(p, 8); }
bool col_ok(const void *p) { return sdb::aligned(p, 16); }

// Natural alignment of every typed pointer (int32/uint32: 4, uint64: 8).  A
// misaligned typed access would fault the device, so the host rejects it.
bool nat4(std::initializer_list<const void *> ps)
{
    for (auto p : ps)
        if (!sdb::aligned(p, 4)) return false;
    return true;
}
bool nat8(const void *p) { return sdb::aligned(p, 8); }
#define SDB_REQUIRE_ALIGNED(cond, what) \
    if (!(cond)) return sdb_set_error(SDB_ERR_INVALID, "%s: pointer not naturally aligned", what)

}  // namespace

// ============================================================== C ABI
namespace {
// The compaction's launches (count_first: the tiles' counts too, else they are
// there from an earlier call over the same flags).
void launch_compact(Compact &a, bool occ, bool count_first, cudaStream_t s)
{
    // lists of 4096 rows up to 4 M rows, so that a middling segment has blocks
    // enough (437,500 slots, 27 blocks of 16384: 14.1 us for the two
    // launches, 107 of 4096: 9.6)
    a.steps = a.n <= (1ull << 22) ? 1 : 4;
    const uint64_t list_rows = (uint64_t)a.steps * kCompactChunk;
    const uint64_t lists = (a.n + list_rows - 1) / list_rows;
    a.subs = (uint32_t)((lists + kCompactTiles - 1) / kCompactTiles);
    const unsigned tiles = (unsigned)((lists + a.subs - 1) / a.subs);
    if (occ) {
        if (count_first) k_compact_count<uint32_t><<<tiles, kThreads, 0, s>>>(a);
        k_compact_write<uint32_t><<<tiles, kThreads, 0, s>>>(a);
    } else {
        if (count_first) k_compact_count<uint8_t><<<tiles, kThreads, 0, s>>>(a);
        k_compact_write<uint8_t><<<tiles, kThreads, 0, s>>>(a);
    }
}
}  // namespace

extern "C" {

int sdb_fill_u8(uint8_t *flags, uint64_t n, uint8_t v, sdb_stream_t stream)
{
    if (n && !flags) return sdb_set_error(SDB_ERR_INVALID, "sdb_fill_u8: NULL buffer");
    return launch_map(n, flags_ok(flags), FillU8{flags, v}, (cudaStream_t)stream, "sdb_fill_u8", SDB_OPK_FILL_U8);
}

int sdb_select_lit(const int32_t *col, int32_t v, int cmp_op, int logic_op, const uint8_t *in, uint8_t *out,
                   uint64_t n, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({col}), "sdb_select_lit");
    if (n && (!col || !in || !out)) return sdb_set_error(SDB_ERR_INVALID, "sdb_select_lit: NULL buffer");
    bool vec = col_ok(col) && flags_ok(in) && flags_ok(out);
    return launch_map(n, vec, SelectLit{col, v, cmp_op, logic_op, in, out}, (cudaStream_t)stream, "sdb_select_lit", SDB_OPK_SELECT_LIT);
}

int sdb_select_cols(const int32_t *a, const int32_t *b, int cmp_op, int logic_op, const uint8_t *in, uint8_t *out,
                    uint64_t n, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({a, b}), "sdb_select_cols");
    if (n && (!a || !b || !in || !out)) return sdb_set_error(SDB_ERR_INVALID, "sdb_select_cols: NULL buffer");
    bool vec = col_ok(a) && col_ok(b) && flags_ok(in) && flags_ok(out);
    return launch_map(n, vec, SelectCols{a, b, cmp_op, logic_op, in, out}, (cudaStream_t)stream, "sdb_select_cols", SDB_OPK_SELECT_COLS);
}

int sdb_logical(int logic_op, const uint8_t *in, const uint8_t *local, uint8_t *out, uint64_t n, sdb_stream_t stream)
{
    if (n && (!in || !local || !out)) return sdb_set_error(SDB_ERR_INVALID, "sdb_logical: NULL buffer");
    bool vec = flags_ok(in) && flags_ok(local) && flags_ok(out);
    return launch_map(n, vec, Logical{logic_op, in, local, out}, (cudaStream_t)stream, "sdb_logical", SDB_OPK_LOGICAL);
}

int sdb_fill_i32(int32_t *dst, int32_t v, uint64_t n, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({dst}), "sdb_fill_i32");
    if (n && !dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_fill_i32: NULL buffer");
    return launch_map(n, col_ok(dst), FillI32{dst, v}, (cudaStream_t)stream, "sdb_fill_i32", SDB_OPK_FILL_I32);
}

static int binop_common(int32_t *res, const int32_t *a, const int32_t *b, int32_t la, int32_t lb, int op, int mode,
                        const uint8_t *flags, uint64_t n, sdb_stream_t stream, const char *what)
{
    SDB_REQUIRE_ALIGNED(nat4({res, a, b}), what);
    if (op < SDB_MUL || op > SDB_SUB) return sdb_set_error(SDB_ERR_INVALID, "%s: unknown operation %d", what, op);
    if (n && (!res || !flags || (mode != 1 && !a) || (mode != 2 && !b)))
        return sdb_set_error(SDB_ERR_INVALID, "%s: NULL buffer", what);
    bool vec = col_ok(res) && col_ok(a) && col_ok(b) && flags_ok(flags);
    return launch_map(n, vec, Binop{res, a, b, la, lb, op, mode, flags}, (cudaStream_t)stream, what, SDB_OPK_BINOP);
}

int sdb_binop_cc(int32_t *res, const int32_t *a, const int32_t *b, int bin_op, const uint8_t *flags, uint64_t n,
                 sdb_stream_t stream)
{
    return binop_common(res, a, b, 0, 0, bin_op, 0, flags, n, stream, "sdb_binop_cc");
}

int sdb_binop_lc(int32_t *res, int32_t a, const int32_t *b, int bin_op, const uint8_t *flags, uint64_t n,
                 sdb_stream_t stream)
{
    return binop_common(res, nullptr, b, a, 0, bin_op, 1, flags, n, stream, "sdb_binop_lc");
}

int sdb_binop_cl(int32_t *res, const int32_t *a, int32_t b, int bin_op, const uint8_t *flags, uint64_t n,
                 sdb_stream_t stream)
{
    return binop_common(res, a, nullptr, 0, b, bin_op, 2, flags, n, stream, "sdb_binop_cl");
}

int sdb_sum_i32_u64(const int32_t *col, const uint8_t *flags, uint64_t n, uint64_t *acc, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({col}) && nat8(acc), "sdb_sum_i32_u64");
    if (!acc || (n && (!col || !flags))) return sdb_set_error(SDB_ERR_INVALID, "sdb_sum_i32_u64: NULL buffer");
    if (n == 0) return SDB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const LaunchShape sh = op_shape(SDB_OPK_SUM, n, 4);
    if (col_ok(col) && flags_ok(flags))
        k_sum<true><<<grid_of((n + 7) / 8, sh), sh.block, 0, s>>>(col, flags, n, acc);
    else
        k_sum<false><<<grid_of(n, sh), sh.block, 0, s>>>(col, flags, n, acc);
    return sdb_check_launch("sdb_sum_i32_u64");
}

int sdb_count_flags(const uint8_t *flags, uint64_t n, uint64_t *out, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat8(out), "sdb_count_flags");
    if (!out || (n && !flags)) return sdb_set_error(SDB_ERR_INVALID, "sdb_count_flags: NULL buffer");
    cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemsetAsync(out, 0, sizeof(uint64_t), s) != cudaSuccess) return sdb_check_launch("sdb_count_flags");
    if (n == 0) return SDB_OK;
    const LaunchShape sh = op_shape(SDB_OPK_COUNT_FLAGS, n, 4);
    if (flags_ok(flags))
        k_count<true><<<grid_of((n + 7) / 8, sh), sh.block, 0, s>>>(flags, n, out);
    else
        k_count<false><<<grid_of(n, sh), sh.block, 0, s>>>(flags, n, out);
    return sdb_check_launch("sdb_count_flags");
}

int sdb_min_max_i32(const int32_t *col, uint64_t n, int32_t *minmax, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({col, minmax}), "sdb_min_max_i32");
    if (n == 0 || !col || !minmax) return sdb_set_error(SDB_ERR_INVALID, "sdb_min_max_i32: empty column or NULL buffer");
    cudaStream_t s = (cudaStream_t)stream;
    k_minmax_init<<<1, 1, 0, s>>>(minmax);
    const LaunchShape sh = op_shape(SDB_OPK_MIN_MAX, n, 4);
    if (col_ok(col))
        k_minmax<true><<<grid_of((n + 7) / 8, sh), sh.block, 0, s>>>(col, n, minmax);
    else
        k_minmax<false><<<grid_of(n, sh), sh.block, 0, s>>>(col, n, minmax);
    sdb_count_launches(1);
    return sdb_check_launch("sdb_min_max_i32");
}

int sdb_groupby_sum(const int32_t *const *keys, const int32_t *mins, const int32_t *maxs, int g, const int32_t *val,
                    const uint8_t *flags, uint64_t n, uint64_t P, int32_t *const *out_keys, uint64_t *out_sum,
                    uint32_t *occ, sdb_stream_t stream)
{
    if (g < 1 || g > 8) return sdb_set_error(SDB_ERR_INVALID, "sdb_groupby_sum: g=%d outside [1,8]", g);
    if (!keys || !mins || !maxs || !out_keys) return sdb_set_error(SDB_ERR_INVALID, "sdb_groupby_sum: NULL host array");
    if (P == 0) return sdb_set_error(SDB_ERR_INVALID, "sdb_groupby_sum: P == 0");
    if (n && (!val || !flags || !out_sum || !occ)) return sdb_set_error(SDB_ERR_INVALID, "sdb_groupby_sum: NULL buffer");
    SDB_REQUIRE_ALIGNED(nat4({val, occ}) && nat8(out_sum), "sdb_groupby_sum");
    for (int j = 0; j < g; j++) SDB_REQUIRE_ALIGNED(nat4({keys[j], out_keys[j]}), "sdb_groupby_sum");
    GroupArgs a{};
    uint32_t mult = 1;
    for (int j = 0; j < g; j++) {
        if (n && (!keys[j] || !out_keys[j])) return sdb_set_error(SDB_ERR_INVALID, "sdb_groupby_sum: NULL key column");
        a.keys[j] = keys[j];
        a.out_keys[j] = out_keys[j];
        a.mins[j] = mins[j];
        a.mults[j] = mult;
        mult *= (uint32_t)maxs[j] - (uint32_t)mins[j] + 1u;
    }
    a.g = g; a.val = val; a.flags = flags; a.n = n; a.P = P; a.out_sum = out_sum; a.occ = occ;
    if (n == 0) return SDB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    // the slot table (P <= 8192: 12 B per slot)
    const size_t smem = P <= 8192 ? (size_t)P * 3 * sizeof(uint32_t) : 0;
    const bool vec = sdb::aligned(flags, 16);
    static sdb::SmemLimit smem_limit;
    smem_limit.allow(8192 * 12, k_groupby_listed<true, true>, k_groupby_listed<true, false>, k_groupby_queued<true>,
                     k_groupby_queued<false>);
    const uint64_t sms = (uint64_t)sdb::device_sms();
    const uint64_t chunks = (n + 511) / 512;  // one per warp at a time
    auto blocks = [&](int threads, uint64_t per_sm) {
        return (unsigned)std::min<uint64_t>((chunks * 32 + threads - 1) / threads, sms * per_sm);
    };
    if (P > 8192) {
        (vec ? k_groupby_listed<false, true> : k_groupby_listed<false, false>)<<<blocks(kThreads, 8), kThreads, 0, s>>>(a);
    } else if (chunks * 32 < sms * kGroupThreads) {
        (vec ? k_groupby_listed<true, true> : k_groupby_listed<true, false>)<<<blocks(kThreads, 2), kThreads, smem, s>>>(a);
    } else {
        (vec ? k_groupby_queued<true> : k_groupby_queued<false>)<<<blocks(kGroupThreads, 2), kGroupThreads, smem, s>>>(a);
    }
    return sdb_check_launch("sdb_groupby_sum");
}

int sdb_occ_to_flags(const uint32_t *occ, uint8_t *flags, uint64_t P, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({occ}), "sdb_occ_to_flags");
    if (P && (!occ || !flags)) return sdb_set_error(SDB_ERR_INVALID, "sdb_occ_to_flags: NULL buffer");
    return launch_map(P, col_ok(occ) && flags_ok(flags), OccToFlags{occ, flags}, (cudaStream_t)stream,
                      "sdb_occ_to_flags", SDB_OPK_OCC_TO_FLAGS);
}

int sdb_ht_build_keys(const int32_t *key, const uint8_t *flags, uint64_t n, uint8_t *ht, int32_t min, int32_t len,
                      sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key}), "sdb_ht_build_keys");
    if (n && (!key || !flags || !ht)) return sdb_set_error(SDB_ERR_INVALID, "sdb_ht_build_keys: NULL buffer");
    if (n == 0) return SDB_OK;
    const LaunchShape sh = op_shape(SDB_OPK_BUILD_KEYS, n, 8);
    k_build_keys<<<grid_of(n, sh), sh.block, 0, (cudaStream_t)stream>>>(key, flags, n, ht, min, len);
    return sdb_check_launch("sdb_ht_build_keys");
}

int sdb_probe_semi(const int32_t *key, const uint8_t *in, uint8_t *out, uint64_t n, const uint8_t *ht, int32_t min,
                   int32_t max, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key}), "sdb_probe_semi");
    if (n && (!key || !in || !out || !ht)) return sdb_set_error(SDB_ERR_INVALID, "sdb_probe_semi: NULL buffer");
    bool vec = col_ok(key) && flags_ok(in) && flags_ok(out);
    return launch_map(n, vec, ProbeSemi{key, in, out, ht, min, max}, (cudaStream_t)stream, "sdb_probe_semi", SDB_OPK_PROBE_SEMI);
}

int sdb_ht_build_kv(const int32_t *key, const int32_t *val, const uint8_t *flags, uint64_t n, int32_t *ht2,
                    int32_t min, int32_t len, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key, val, ht2}), "sdb_ht_build_kv");
    if (n && (!key || !val || !flags || !ht2)) return sdb_set_error(SDB_ERR_INVALID, "sdb_ht_build_kv: NULL buffer");
    if (n == 0) return SDB_OK;
    const LaunchShape sh = op_shape(SDB_OPK_BUILD_KV, n, 8);
    k_build_kv<<<grid_of(n, sh), sh.block, 0, (cudaStream_t)stream>>>(key, val, flags, n, ht2, min, len);
    return sdb_check_launch("sdb_ht_build_kv");
}

int sdb_probe_full(const int32_t *key, int32_t *val_out, const uint8_t *in, uint8_t *out, uint64_t n,
                   const int32_t *ht2, int32_t min, int32_t max, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key, val_out, ht2}), "sdb_probe_full");
    if (n && (!key || !val_out || !in || !out || !ht2))
        return sdb_set_error(SDB_ERR_INVALID, "sdb_probe_full: NULL buffer");
    bool vec = col_ok(key) && flags_ok(in) && flags_ok(out);
    cudaStream_t s = (cudaStream_t)stream;
    if (sdb::aligned(ht2, 8))
        return launch_map(n, vec, ProbeFull<true>{key, val_out, in, out, ht2, min, max}, s, "sdb_probe_full", SDB_OPK_PROBE_FULL);
    return launch_map(n, vec, ProbeFull<false>{key, val_out, in, out, ht2, min, max}, s, "sdb_probe_full", SDB_OPK_PROBE_FULL);
}

int sdb_oa_log2_slots(uint64_t build_rows)
{
    if (build_rows > (1ull << 30)) return sdb_set_error(SDB_ERR_INVALID, "sdb_oa_log2_slots: more than 2^30 rows");
    int lg = 4;
    while ((1ull << lg) < 2 * build_rows) lg++;
    return lg;
}

// Checks the arguments every open-addressing entry shares.
static int oa_check(const char *what, int lg, int32_t mn, int32_t mx, const void *ht, uintptr_t align)
{
    if (lg < 1 || lg > 31) return sdb_set_error(SDB_ERR_INVALID, "%s: log2_slots=%d outside [1,31]", what, lg);
    if (mn > mx || (uint32_t)mx - (uint32_t)mn >= 0x7fffffffu)
        return sdb_set_error(SDB_ERR_INVALID, "%s: key range [%d,%d] empty or 2^31 keys or more", what, mn, mx);
    if (!sdb::aligned(ht, align)) return sdb_set_error(SDB_ERR_INVALID, "%s: table not %d-byte aligned", what, (int)align);
    return SDB_OK;
}

int sdb_ht_build_keys_oa(const int32_t *key, const uint8_t *flags, uint64_t n, uint32_t *ht, int log2_slots,
                         int32_t min, int32_t max, int fresh, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key}), "sdb_ht_build_keys_oa");
    if (n && (!key || !flags || !ht)) return sdb_set_error(SDB_ERR_INVALID, "sdb_ht_build_keys_oa: NULL buffer");
    int st = oa_check("sdb_ht_build_keys_oa", log2_slots, min, max, ht, 4);
    if (st != SDB_OK || n == 0) return st;
    const LaunchShape sh = op_shape(SDB_OPK_BUILD_KEYS, n, 8);
    k_build_keys_oa<<<grid_of(n, sh), sh.block, 0, (cudaStream_t)stream>>>(key, flags, n, ht, log2_slots, min, max,
                                                                          fresh);
    return sdb_check_launch("sdb_ht_build_keys_oa");
}

int sdb_probe_semi_oa(const int32_t *key, const uint8_t *in, uint8_t *out, uint64_t n, const uint32_t *ht,
                      int log2_slots, int32_t min, int32_t max, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key}), "sdb_probe_semi_oa");
    if (n && (!key || !in || !out || !ht)) return sdb_set_error(SDB_ERR_INVALID, "sdb_probe_semi_oa: NULL buffer");
    int st = oa_check("sdb_probe_semi_oa", log2_slots, min, max, ht, 4);
    if (st != SDB_OK) return st;
    bool vec = col_ok(key) && flags_ok(in) && flags_ok(out);
    return launch_map(n, vec, ProbeSemiOA{key, in, out, ht, log2_slots, min, max}, (cudaStream_t)stream,
                      "sdb_probe_semi_oa", SDB_OPK_PROBE_SEMI);
}

int sdb_ht_build_kv_oa(const int32_t *key, const int32_t *val, const uint8_t *flags, uint64_t n, int32_t *ht2,
                       int log2_slots, int32_t min, int32_t max, int fresh, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key, val}), "sdb_ht_build_kv_oa");
    if (n && (!key || !val || !flags || !ht2)) return sdb_set_error(SDB_ERR_INVALID, "sdb_ht_build_kv_oa: NULL buffer");
    int st = oa_check("sdb_ht_build_kv_oa", log2_slots, min, max, ht2, 8);
    if (st != SDB_OK || n == 0) return st;
    const LaunchShape sh = op_shape(SDB_OPK_BUILD_KV, n, 8);
    k_build_kv_oa<<<grid_of(n, sh), sh.block, 0, (cudaStream_t)stream>>>(key, val, flags, n, ht2, log2_slots, min,
                                                                        max, fresh);
    return sdb_check_launch("sdb_ht_build_kv_oa");
}

int sdb_probe_full_oa(const int32_t *key, int32_t *val_out, const uint8_t *in, uint8_t *out, uint64_t n,
                      const int32_t *ht2, int log2_slots, int32_t min, int32_t max, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({key, val_out}), "sdb_probe_full_oa");
    if (n && (!key || !val_out || !in || !out || !ht2))
        return sdb_set_error(SDB_ERR_INVALID, "sdb_probe_full_oa: NULL buffer");
    int st = oa_check("sdb_probe_full_oa", log2_slots, min, max, ht2, 8);
    if (st != SDB_OK) return st;
    bool vec = col_ok(key) && flags_ok(in) && flags_ok(out);
    return launch_map(n, vec, ProbeFullOA{key, val_out, in, out, ht2, log2_slots, min, max}, (cudaStream_t)stream,
                      "sdb_probe_full_oa", SDB_OPK_PROBE_FULL);
}

size_t sdb_compact_scratch_bytes(uint64_t n)
{
    uint64_t nchunks = (n + kCompactChunk - 1) / kCompactChunk;
    return (size_t)((nchunks * sizeof(uint32_t) + 255) & ~(uint64_t)255);
}

int sdb_compact_row_ids(const uint8_t *flags, uint64_t n, int32_t *ids, uint32_t *count, void *scratch,
                        size_t scratch_bytes, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({ids, count, scratch}), "sdb_compact_row_ids");
    if (!count) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_row_ids: NULL count");
    if (n > (uint64_t)INT32_MAX + 1) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_row_ids: n too large for int32 ids");
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) {
        if (cudaMemsetAsync(count, 0, sizeof(uint32_t), s) != cudaSuccess) return sdb_check_launch("sdb_compact_row_ids");
        return SDB_OK;
    }
    if (!flags || !ids) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_row_ids: NULL buffer");
    if (!sdb::aligned(flags, 16)) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_row_ids: flags must be 16-byte aligned");
    if (!scratch || scratch_bytes < sdb_compact_scratch_bytes(n))
        return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_row_ids: scratch needs %zu bytes", sdb_compact_scratch_bytes(n));
    Compact a{};
    a.flags = flags;
    a.n = n;
    a.counts = static_cast<uint32_t *>(scratch);
    a.ids = ids;
    a.count = count;
    launch_compact(a, false, true, s);
    sdb_count_launches(1);
    return sdb_check_launch("sdb_compact_row_ids");
}

}  // extern "C"

// ---------------------------------------------------------------- no-allocation compaction
// Scratch of sdb_compact_row_ids_noalloc: the per-chunk counts for one
// segment of up to SDB_COMPACT_NOALLOC_MAX_ROWS rows (256 KB).  It lives in
// the library's own device image, so every device that loads the library
// holds it until the process exits, and every call on that device shares it.
static_assert(SDB_COMPACT_NOALLOC_MAX_ROWS % kCompactChunk == 0,
              "the no-allocation scratch holds one count per whole chunk of the largest segment");
static __device__ __align__(256) uint32_t g_noalloc_compact_scratch[SDB_COMPACT_NOALLOC_MAX_ROWS / kCompactChunk];
// what sdb_compact_scratch_bytes(SDB_COMPACT_NOALLOC_MAX_ROWS) asks for must fit the array
static_assert(((SDB_COMPACT_NOALLOC_MAX_ROWS / kCompactChunk) * sizeof(uint32_t) + 255) / 256 * 256 <=
                  sizeof(g_noalloc_compact_scratch),
              "no-allocation scratch smaller than the compaction needs at the row limit");

namespace {
constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void *g_noalloc_scratch_ptr[kNoAllocMaxDevices];  // device address of the array, per device (set up once)
}  // namespace

extern "C" {

int sdb_compact_row_ids_noalloc(const uint8_t *flags, uint64_t n, int32_t *ids, uint32_t *count, sdb_stream_t stream)
{
    if (n > SDB_COMPACT_NOALLOC_MAX_ROWS)
        return sdb_set_error(SDB_ERR_INVALID,
                             "sdb_compact_row_ids_noalloc: %llu rows exceed the fixed scratch (at most %llu rows per call)",
                             (unsigned long long)n, (unsigned long long)SDB_COMPACT_NOALLOC_MAX_ROWS);
    if (n == 0) return sdb_compact_row_ids(flags, 0, ids, count, nullptr, 0, stream);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return sdb_set_error(SDB_ERR_CUDA, "sdb_compact_row_ids_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_row_ids_noalloc: device %d beyond the supported %d", dev,
                             kNoAllocMaxDevices);
    void *scratch = nullptr;
    {
        // Set-up, once per device, with that device current: the host-side
        // name of the array is not a device address, so ask the runtime for it.
        // The address is kept for the life of the process; a cudaDeviceReset
        // destroys the module that holds the array, so the entry must not be
        // called on a device after it was reset.
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_scratch_ptr[dev]) {
            void *p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_compact_scratch);
            if (e != cudaSuccess || !p)
                return sdb_set_error(SDB_ERR_CUDA, "sdb_compact_row_ids_noalloc: cudaGetSymbolAddress: %s",
                                     cudaGetErrorString(e));
            g_noalloc_scratch_ptr[dev] = p;
        }
        scratch = g_noalloc_scratch_ptr[dev];
    }
    // Every count the passes read is written first by k_compact_count, so the
    // array needs no clearing between calls.
    return sdb_compact_row_ids(flags, n, ids, count, scratch, sizeof(g_noalloc_compact_scratch), stream);
}

static int compact_gather(const void *flags, bool occ, uint64_t n, int ncols, const void *const *src, const int *wide,
                          void *const *dst, uint32_t *count, sdb_stream_t stream)
{
    if (n > kSmallCompactMax) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather: n=%llu exceeds %u",
                                                   (unsigned long long)n, kSmallCompactMax);
    if (ncols < 0 || ncols > kCompactCols || (ncols && (!src || !wide || !dst)))
        return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather: 0..%d columns", kCompactCols);
    if (!count || (n && !flags)) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather: NULL flags or count");
    if (occ && !sdb::aligned(flags, 4)) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather_occ: occ misaligned");
    if (!sdb::aligned(count, 4)) return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather: count misaligned");
    Compact a{};
    a.flags = flags;
    a.n = n;
    a.ncols = ncols;
    a.count = count;
    for (int c = 0; c < ncols; c++) {
        const size_t w = wide[c] ? 8 : 4;
        if (!src[c] || !dst[c] || !sdb::aligned(src[c], w) || !sdb::aligned(dst[c], w))
            return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather: column %d NULL or misaligned", c);
        a.src[c] = src[c];
        a.dst[c] = dst[c];
        a.wide[c] = wide[c] ? 1 : 0;
    }
    const unsigned blocks = (unsigned)std::max<uint64_t>(1, (n + 4 * kSmallCompactThreads - 1) / (4 * kSmallCompactThreads));
    const bool vec = sdb::aligned(flags, occ ? 16 : 4);
    auto kern = occ ? (vec ? k_compact_gather_small<uint32_t, true> : k_compact_gather_small<uint32_t, false>)
                    : (vec ? k_compact_gather_small<uint8_t, true> : k_compact_gather_small<uint8_t, false>);
    kern<<<blocks, kSmallCompactThreads, 0, (cudaStream_t)stream>>>(a);
    return sdb_check_launch("sdb_compact_gather");
}

int sdb_compact_gather(const uint8_t *flags, uint64_t n, int ncols, const void *const *src, const int *wide,
                       void *const *dst, uint32_t *count, sdb_stream_t stream)
{
    return compact_gather(flags, false, n, ncols, src, wide, dst, count, stream);
}

int sdb_compact_gather_occ(const uint32_t *occ, uint64_t n, int ncols, const void *const *src, const int *wide,
                           void *const *dst, uint32_t *count, sdb_stream_t stream)
{
    return compact_gather(occ, true, n, ncols, src, wide, dst, count, stream);
}

int sdb_gather_i32(const int32_t *src, const int32_t *ids, const uint32_t *count, int32_t *dst, uint64_t cap,
                   sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({src, ids, count, dst}), "sdb_gather_i32");
    if (cap == 0) return SDB_OK;
    if (!src || !ids || !count || !dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gather_i32: NULL buffer");
    const LaunchShape sh = op_shape(SDB_OPK_GATHER, cap, 8);
    k_gather<int32_t><<<grid_of(cap, sh), sh.block, 0, (cudaStream_t)stream>>>(src, ids, count, dst, cap);
    return sdb_check_launch("sdb_gather_i32");
}

int sdb_gather_u64(const uint64_t *src, const int32_t *ids, const uint32_t *count, uint64_t *dst, uint64_t cap,
                   sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({ids, count}) && nat8(src) && nat8(dst), "sdb_gather_u64");
    if (cap == 0) return SDB_OK;
    if (!src || !ids || !count || !dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gather_u64: NULL buffer");
    const LaunchShape sh = op_shape(SDB_OPK_GATHER, cap, 8);
    k_gather<uint64_t><<<grid_of(cap, sh), sh.block, 0, (cudaStream_t)stream>>>(src, ids, count, dst, cap);
    return sdb_check_launch("sdb_gather_u64");
}

int32_t sdb_gen_uniform_host(uint64_t seed, uint64_t stream_id, uint64_t row, int32_t lo, int32_t hi)
{
    return sdb::uniform_from_key(sdb::stream_key(seed, stream_id), row, lo, hi);
}

int sdb_gen_uniform(int32_t *dst, uint64_t n, uint64_t row0, uint64_t seed, uint64_t stream_id, int32_t lo,
                    int32_t hi, sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({dst}), "sdb_gen_uniform");
    if (hi < lo) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_uniform: hi < lo");
    if (n == 0) return SDB_OK;
    if (!dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_uniform: NULL buffer");
    k_gen_uniform<<<sdb::grid_for(n, kThreads), kThreads, 0, (cudaStream_t)stream>>>(
        dst, n, row0, sdb::stream_key(seed, stream_id), lo, hi);
    return sdb_check_launch("sdb_gen_uniform");
}

int sdb_gen_uniform_cpu(int32_t *dst, uint64_t n, uint64_t row0, uint64_t seed, uint64_t stream_id, int32_t lo,
                        int32_t hi)
{
    if (hi < lo) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_uniform_cpu: hi < lo");
    if (n && !dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_uniform_cpu: NULL buffer");
    const uint64_t key = sdb::stream_key(seed, stream_id);
    parallel_rows(n, [=](uint64_t i) { dst[i] = sdb::uniform_from_key(key, row0 + i, lo, hi); });
    return SDB_OK;
}

int sdb_gen_datekeys_cpu(int32_t *dst, uint64_t n, int64_t day0)
{
    if (n && !dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_datekeys_cpu: NULL buffer");
    for (uint64_t i = 0; i < n; i++) dst[i] = sdb::datekey_of_day(day0 + (int64_t)i);
    return SDB_OK;
}

int sdb_gen_dates(int32_t *dst, uint64_t n, uint64_t row0, uint64_t seed, uint64_t stream_id, int32_t ndays,
                  sdb_stream_t stream)
{
    SDB_REQUIRE_ALIGNED(nat4({dst}), "sdb_gen_dates");
    if (ndays < 1) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_dates: ndays < 1");
    if (n == 0) return SDB_OK;
    if (!dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_dates: NULL buffer");
    k_gen_dates<<<sdb::grid_for(n, kThreads), kThreads, 0, (cudaStream_t)stream>>>(
        dst, n, row0, sdb::stream_key(seed, stream_id), ndays);
    return sdb_check_launch("sdb_gen_dates");
}

int sdb_gen_dates_cpu(int32_t *dst, uint64_t n, uint64_t row0, uint64_t seed, uint64_t stream_id, int32_t ndays)
{
    if (ndays < 1) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_dates_cpu: ndays < 1");
    if (n && !dst) return sdb_set_error(SDB_ERR_INVALID, "sdb_gen_dates_cpu: NULL buffer");
    const uint64_t key = sdb::stream_key(seed, stream_id);
    parallel_rows(n, [=](uint64_t i) { dst[i] = sdb::datekey_of_day(sdb::uniform_from_key(key, row0 + i, 0, ndays - 1)); });
    return SDB_OK;
}

}  // extern "C"

extern "C" {

int sdb_op_tune_set(int op_kernel, uint64_t rows, int block, int blocks_per_sm)
{
    if (op_kernel < 0 || op_kernel >= SDB_OPK_COUNT) return sdb_set_error(SDB_ERR_INVALID, "sdb_op_tune_set: bad kernel");
    int32_t e = 0;
    if (block != 0 || blocks_per_sm != 0) {
        if (block != 128 && block != 256 && block != 512)
            return sdb_set_error(SDB_ERR_INVALID, "sdb_op_tune_set: block must be 128, 256 or 512");
        if (blocks_per_sm < 1 || blocks_per_sm > 32 || blocks_per_sm * block > 2048)
            return sdb_set_error(SDB_ERR_INVALID, "sdb_op_tune_set: blocks_per_sm must be 1..32 and fit 2048 threads");
        e = (block << 8) | blocks_per_sm;
    }
    g_op_tune[op_kernel][op_bucket(rows)].store(e, std::memory_order_relaxed);
    return SDB_OK;
}

int sdb_op_tune_get(int op_kernel, uint64_t rows, int *block, int *blocks_per_sm)
{
    if (op_kernel < 0 || op_kernel >= SDB_OPK_COUNT || !block || !blocks_per_sm)
        return sdb_set_error(SDB_ERR_INVALID, "sdb_op_tune_get: bad argument");
    const int def = (op_kernel == SDB_OPK_SUM || op_kernel == SDB_OPK_COUNT_FLAGS || op_kernel == SDB_OPK_MIN_MAX) ? 4 : 8;
    const LaunchShape sh = op_shape(op_kernel, rows, def);
    *block = sh.block;
    *blocks_per_sm = sh.per_sm;
    return SDB_OK;
}

}  // extern "C"

namespace {
// Every row of a segment (a result no filter applies to, a scalar sum): what
// the compaction gives for flags that are all true, without flags.
__global__ void __launch_bounds__(kThreads) k_copy_rows(const __grid_constant__ Compact a)
{
    const uint64_t stride = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i = blockIdx.x * (uint64_t)kThreads + threadIdx.x; i < a.n; i += stride)
        for (int c = 0; c < a.ncols; c++) {
            if (a.wide[c]) static_cast<uint64_t *>(a.dst[c])[i] = static_cast<const uint64_t *>(a.src[c])[i];
            else static_cast<int32_t *>(a.dst[c])[i] = static_cast<const int32_t *>(a.src[c])[i];
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.count = (uint32_t)a.n;
}

constexpr uint64_t kMaxResultSegment = 1ull << 31;  // as sdb_compact_row_ids: row numbers and counts fit their words
}  // namespace

// All rows of a segment (at most 2^31) copied from up to 8 columns.
int sdb_copy_rows(uint64_t n, int ncols, const void *const *src, const int *wide, void *const *dst, uint32_t *count,
                  cudaStream_t s)
{
    if (ncols > kCompactCols) return sdb_set_error(SDB_ERR_INVALID, "sdb_copy_rows: at most %d columns", kCompactCols);
    if (n > kMaxResultSegment) return sdb_set_error(SDB_ERR_INVALID, "sdb_copy_rows: a segment of more than 2^31 rows");
    Compact a{};
    a.n = n;
    a.ncols = ncols;
    a.count = count;
    for (int c = 0; c < ncols; c++) {
        a.src[c] = src[c];
        a.dst[c] = dst[c];
        a.wide[c] = wide[c];
    }
    k_copy_rows<<<sdb::grid_for(n, kThreads, 8), kThreads, 0, s>>>(a);
    return sdb_check_launch("sdb_copy_rows");
}

// The flagged rows of a segment of 1 to 2^31 rows (flags or occupancy words,
// 16-byte aligned) gathered from any number of columns: what sdb_compact_row_ids
// and one sdb_gather_* per column give together.  Scratch as for
// sdb_compact_row_ids.  For the executor's results above sdb_compact_gather's
// limits.
int sdb_compact_gather_large(const void *flags, bool occ, uint64_t n, int ncols, const void *const *src, const int *wide,
                             void *const *dst, uint32_t *count, void *scratch, cudaStream_t s)
{
    if (n == 0 || n > kMaxResultSegment)
        return sdb_set_error(SDB_ERR_INVALID, "sdb_compact_gather_large: a segment of no rows or more than 2^31");
    Compact a{};
    a.flags = flags;
    a.n = n;
    a.counts = static_cast<uint32_t *>(scratch);
    a.count = count;
    int launches = 0;
    for (int c0 = 0; c0 == 0 || c0 < ncols; c0 += kCompactCols) {
        a.ncols = std::min(kCompactCols, ncols - c0);
        for (int c = 0; c < a.ncols; c++) {
            a.src[c] = src[c0 + c];
            a.dst[c] = dst[c0 + c];
            a.wide[c] = wide[c0 + c];
        }
        launch_compact(a, occ, c0 == 0, s);
        launches += c0 == 0 ? 2 : 1;
    }
    sdb_count_launches((unsigned)launches - 1);
    return sdb_check_launch("sdb_compact_gather_large");
}
