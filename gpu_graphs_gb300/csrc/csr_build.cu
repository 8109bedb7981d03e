// csr_build.cu -- on-device edge list -> CSR (sm_103a).
//
// The reference builds CSR on the host: vector<vector<int>> adjacency lists
// filled line by line, then flattened (1D Partition/src/csr.cpp:25-65,
// 2D Partition/src/csc.cpp:18-89), with no dedup, no self-loop removal and
// no symmetrisation.  Here the same CSR (rows sorted, which does not change
// BFS levels) is built in HBM:
//   1. k_count   degree histogram (warp-aggregated atomics: match_any groups
//                lanes with the same source so hubs take one atomic)
//   2. scan      decoupled look-back exclusive scan -> row offsets
//   3. k_scatter each edge to its row (aggregated atomic cursors)
//      Large inputs with ids all over take two steps instead of 1 to 3:
//      k_bucket_scatter sorts the entries into buckets of 1024 rows, then
//      k_bucket_rows lays out one bucket per CTA
//   4. k_bin + per-row sorts by length: up to 32 entries in a warp's registers
//                (k_sort_small), up to 512 (k_sort_warp), up to 4096 in a CTA's
//                (k_sort_block); longer rows through bitmaps of the vertices
//                (k_long_rows, deduplicating builds of up to 4.3 M vertices),
//                else in sorted chunks of 4096 merged pairwise, every chunk of
//                every row in parallel (k_merge);
//                each row also counts (and packs to its front) its distinct
//                values when deduplicating
//   5. scan + k_compact   packed rows -> final col_idx (dedup only)
//   6. k_finalize zero-degree bitmap, max degree, non-isolated count
#include <algorithm>
#include <climits>
#include <cstdio>

#include "common.cuh"
#include "csr_build.cuh"
#include "index.h"
#include "pinned.cuh"
#include "scan.cuh"

namespace gbfs {

static thread_local int tl_route = 0;

int csr_build_route() { return tl_route; }

namespace {

constexpr int W4_MAX = 128;       // rows up to this length: warp sort, 4 values per lane
constexpr int W16_MAX = 512;      // rows up to this length: warp sort, 16 values per lane
constexpr int SB_E = 8;           // values per thread of a CTA sort
constexpr int MED_MAX = 4096;     // rows up to this length: CTA sort; longer ones in chunks of it
constexpr int MED_THREADS = MED_MAX / SB_E;
constexpr int BIN_THREADS = 1024;
// CTAs of the passes over the edge list: more than fit at once, so that what
// neighbouring CTAs write stays close together (RMAT-22 build 10.2 ms with 16
// per SM, 9.7 with 64)
constexpr int EDGE_CTAS = 152 * 64;
// row classes of k_bin: warp sorts, CTA sorts of 1024, 2048 and 4096, long rows
enum BinClass : int { BIN_W4, BIN_W16, BIN_1K, BIN_2K, BIN_4K, BIN_LONG, BIN_CLASSES };

#define NEED_PINNED(slot)                                                        \
    do {                                                                         \
        if (!(slot)) {                                                           \
            err = "pinned memory for results";                                   \
            return GBFS_ERR_OOM;                                                 \
        }                                                                        \
    } while (0)

#define CK(call)                                                                 \
    do {                                                                         \
        cudaError_t e_ = (call);                                                 \
        if (e_ != cudaSuccess) {                                                 \
            cudaGetLastError(); /* or the next call's launches report it */      \
            err = std::string(#call) + ": " + cudaGetErrorString(e_);            \
            rc = (e_ == cudaErrorMemoryAllocation) ? GBFS_ERR_OOM : GBFS_ERR_CUDA; \
            goto done;                                                           \
        }                                                                        \
    } while (0)

__device__ __forceinline__ int atomic_add_t(int *p, int v) { return atomicAdd(p, v); }
__device__ __forceinline__ long long atomic_add_t(long long *p, long long v)
{
    return (long long)atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v);
}

// All 32 lanes call; key < 0 means "no increment".  Returns the old value of
// arr[key] plus this lane's rank among lanes with the same key.  Lanes are
// grouped by key (one atomic per group) only where two lanes beside each other
// have the same one: random keys hardly ever do, a row that many lanes hit does.
template <typename T>
__device__ __forceinline__ T agg_atomic_add(T *arr, int key)
{
    const int beside = __shfl_xor_sync(FULL, key, 1);
    if (!__any_sync(FULL, key >= 0 && key == beside)) return key >= 0 ? atomic_add_t(&arr[key], (T)1) : (T)0;
    unsigned peers = __match_any_sync(FULL, key);
    int leader = __ffs(peers) - 1;
    T old = 0;
    if (key >= 0 && (int)lane_id() == leader) old = atomic_add_t(&arr[key], (T)__popc(peers));
    old = __shfl_sync(FULL, old, leader);
    return old + (T)__popc(peers & lanemask_lt());
}

template <typename T>
__device__ __forceinline__ T block_sum(T x, T *s_red)
{
    x = warp_sum(x);
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) s_red[warp] = x;
    __syncthreads();
    T t = 0;
    if (warp == 0) {
        t = lane < (blockDim.x >> 5) ? s_red[lane] : 0;
        t = warp_sum(t);
    }
    return t;  // valid in thread 0
}

// Exclusive block scan (blockDim.x <= 1024); returns the prefix, *total set.
__device__ __forceinline__ int block_excl_scan(int x, int *s_warp, int *total)
{
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int incl = warp_incl_scan(x);
    __syncthreads();
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nw ? s_warp[lane] : 0;
        int wi = warp_incl_scan(w);
        if (lane < nw) s_warp[lane] = wi - w;
        if (lane == nw - 1) s_warp[32] = wi;
    }
    __syncthreads();
    *total = s_warp[32];
    return s_warp[warp] + incl - x;
}

__global__ void k_count(const int *__restrict__ src, const int *__restrict__ dst, int64_t m,
                        int n, unsigned flags, int *deg, unsigned long long *total, int *status)
{
    __shared__ unsigned long long s_red[32];
    const bool sym = flags & GBFS_SYMMETRIZE, noself = flags & GBFS_DROP_SELF_LOOPS;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    unsigned long long mine = 0;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < m;
         base += stride) {
        int64_t i = base + lane_id();
        int u = -1, v = -1;
        if (i < m) {
            u = src[i];
            v = dst[i];
            if ((unsigned)u >= (unsigned)n || (unsigned)v >= (unsigned)n) {
                atomicExch(status, DEV_BAD_ID);
                u = v = -1;
            } else if (noself && u == v) {
                u = v = -1;
            }
        }
        // (every lane calls agg_atomic_add); a row of 2^30 edges or more
        // would overflow the int32 degrees
        const int cu = agg_atomic_add(deg, u);
        if (u >= 0 && cu >= (1 << 30)) atomicExch(status, DEV_OVERFLOW);
        mine += u >= 0;
        if (sym) {
            const int cv = agg_atomic_add(deg, v);
            if (v >= 0 && cv >= (1 << 30)) atomicExch(status, DEV_OVERFLOW);
            mine += v >= 0;
        }
    }
    unsigned long long t = block_sum(mine, s_red);
    if (threadIdx.x == 0 && t) atomicAdd(total, t);
}

template <typename RT>
__global__ void k_scatter(const int *__restrict__ src, const int *__restrict__ dst, int64_t m,
                          int n, unsigned flags, RT *cursor, int *tmp)
{
    const bool sym = flags & GBFS_SYMMETRIZE, noself = flags & GBFS_DROP_SELF_LOOPS;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < m;
         base += stride) {
        int64_t i = base + lane_id();
        int u = -1, v = -1;
        if (i < m) {
            u = src[i];
            v = dst[i];
            if ((unsigned)u >= (unsigned)n || (unsigned)v >= (unsigned)n || (noself && u == v))
                u = v = -1;
        }
        const RT p = agg_atomic_add(cursor, u);
        if (u >= 0) tmp[p] = v;
        if (sym) {
            const RT q = agg_atomic_add(cursor, v);
            if (v >= 0) tmp[q] = u;
        }
    }
}

// ---- entries by buckets of rows ----
// Scattering a power-law graph's entries straight to their rows writes each
// 32-byte sector of the columns in eight pieces, far apart in time: RMAT-22
// (134 M entries) spent 1.2 ms counting and 2.8 ms scattering, most of it on
// partly written sectors leaving L2.  With buckets of 2^BK_LOG rows in between,
// every write lands beside others of its time: first each entry goes to its
// bucket as one 32-bit word (row within the bucket, column), in runs gathered
// in shared memory; then one CTA per bucket counts its rows in shared memory,
// writes their offsets and places the columns, all within a range that L2 holds.
// For inputs of BK_MIN_M entries (below, the direct scatter's range fits L2: whole
// builds, buckets and direct, RMAT of 8 M entries 0.99 and 0.87 ms, 25 M 1.50 and
// 1.59, 34 M 1.73 and 1.88, 67 M 2.88 and 3.29, 134 M 4.8 and 6.4; uniform random
// of 12 M entries 0.97 and 0.86, 67 M 2.5 and 3.7) on up to BK_MAX_N vertices (a
// word holds 10 + 22 bits), unless one bucket holds more than BK_MAX_BUCKET
// entries, which would be one CTA's tail, or edges beside each other mostly have
// both ends in the same buckets (a grid's in order, 16 M entries: 1.21 and 0.88 ms).
constexpr int BK_LOG = 10;
constexpr int BK_MAX_N = 1 << 22;
constexpr int BK_BUCKETS = BK_MAX_N >> BK_LOG;
constexpr int64_t BK_MIN_M = 20 << 20;
constexpr unsigned BK_MAX_BUCKET = 1 << 20;
constexpr int BK_BLOCK = 1024;
constexpr int BK_ILP = 8;                          // entries per thread in flight in k_bucket_rows
constexpr int BK_STAGE = 48 << 10;                 // entries of a bucket laid out in shared memory
constexpr int BK_EDGES = 8;                        // input edges per thread and tile
constexpr int BK_SBLOCK = 1024;                    // k_bucket_scatter: one CTA per SM
constexpr int BK_TILE = 2 * BK_SBLOCK * BK_EDGES;  // entries per tile at most
constexpr int BK_PER = BK_BUCKETS / BK_SBLOCK;     // buckets per thread there
static_assert(BK_BUCKETS == 4 * BK_BLOCK, "four buckets per thread");

struct BucketPlan {
    unsigned long long total;
    unsigned largest, near;          // near, seen: edges of a sample beside one in the same buckets, and all
    unsigned seen, over;             // over: entries in buckets too large for shared memory, together
    unsigned bigs, others;
    unsigned hist[BK_BUCKETS];       // zeroed by the caller
    int start[BK_BUCKETS + 1];
    int cursor[BK_BUCKETS];
    int order[BK_BUCKETS];           // the large buckets first
    int over_at[BK_BUCKETS];         // of those too large: where in the spare buffer
};

// The input edge i as up to two entries (u -> v, and v -> u with sym); u = -1:
// none.  Ids outside [0, n) are reported.
__device__ __forceinline__ void load_edge(const int *__restrict__ src, const int *__restrict__ dst, int64_t i, int64_t m,
                                          int n, bool noself, int *status, int &u, int &v)
{
    u = v = -1;
    if (i >= m) return;
    u = src[i];
    v = dst[i];
    if ((unsigned)u >= (unsigned)n || (unsigned)v >= (unsigned)n) {
        atomicExch(status, DEV_BAD_ID);
        u = v = -1;
    } else if (noself && u == v) {
        u = v = -1;
    }
}

__global__ void __launch_bounds__(BK_BLOCK)
k_bucket_hist(const int *__restrict__ src, const int *__restrict__ dst, int64_t m, int n, unsigned flags,
              BucketPlan *plan, int *status)
{
    __shared__ unsigned s_hist[BK_BUCKETS];
    const bool sym = flags & GBFS_SYMMETRIZE, noself = flags & GBFS_DROP_SELF_LOOPS;
    for (int b = (int)threadIdx.x; b < BK_BUCKETS; b += BK_BLOCK) s_hist[b] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * BK_BLOCK;
    unsigned near = 0, seen = 0;
    for (int64_t w0 = (int64_t)blockIdx.x * BK_BLOCK + (threadIdx.x & ~31u); w0 < m; w0 += 4 * stride) {
        const int64_t i0 = w0 + lane_id();  // (whole warps go round)
        int u[4], v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) load_edge(src, dst, i0 + q * stride, m, n, noself, status, u[q], v[q]);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (u[q] < 0) continue;
            atomicAdd(&s_hist[u[q] >> BK_LOG], 1u);
            if (sym) atomicAdd(&s_hist[v[q] >> BK_LOG], 1u);
        }
        if (w0 < stride) {  // the sample: the warps' first edges (every lane calls the shuffles)
            const int u1 = __shfl_xor_sync(FULL, u[0], 1), v1 = __shfl_xor_sync(FULL, v[0], 1);
            if (u[0] >= 0) {
                near = (u[0] ^ u1) >> BK_LOG == 0 && (v[0] ^ v1) >> BK_LOG == 0;
                seen = 1;
            }
        }
    }
    __syncthreads();
    for (int b = (int)threadIdx.x; b < BK_BUCKETS; b += BK_BLOCK)
        if (s_hist[b]) atomicAdd(&plan->hist[b], s_hist[b]);
    near = warp_sum(near);
    seen = warp_sum(seen);
    if (lane_id() == 0) {
        atomicAdd(&plan->near, near);
        atomicAdd(&plan->seen, seen);
    }
}

// One CTA: where each bucket starts, the largest, and the order to lay them out.
__global__ void __launch_bounds__(BK_BLOCK) k_bucket_plan(BucketPlan *plan, int nb)
{
    __shared__ int s_warp[33];
    const int b0 = 4 * (int)threadIdx.x;
    int c[4], sum = 0, most = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        c[k] = (int)plan->hist[b0 + k];
        sum += c[k];
        most = max(most, c[k]);
    }
    int total;
    int at = block_excl_scan(sum, s_warp, &total);
    if (threadIdx.x == 0) {
        plan->total = (unsigned long long)total;
        plan->start[BK_BUCKETS] = total;
    }
    atomicMax(&plan->largest, (unsigned)most);
    int mine_over = 0, over;
#pragma unroll
    for (int k = 0; k < 4; k++) mine_over += c[k] > BK_STAGE ? c[k] : 0;
    int over_at = block_excl_scan(mine_over, s_warp, &over);
    if (threadIdx.x == 0) plan->over = (unsigned)over;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        plan->over_at[b0 + k] = over_at;
        over_at += c[k] > BK_STAGE ? c[k] : 0;
    }
    const long long big = 2ll * (total / nb) + 1;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        plan->start[b0 + k] = at;
        plan->cursor[b0 + k] = at;
        at += c[k];
        if (b0 + k >= nb) continue;
        const int pos = c[k] >= big ? (int)atomicAdd(&plan->bigs, 1u) : nb - 1 - (int)atomicAdd(&plan->others, 1u);
        plan->order[pos] = b0 + k;
    }
}

struct BucketShared {
    int2 run[BK_BUCKETS];   // x: entries of the bucket in the tile, then where its run starts there; y: and in the output
    uint2 entry[BK_TILE];   // the runs: word, place in the output
    int warp[33];
};

__global__ void __launch_bounds__(BK_SBLOCK, 1)
k_bucket_scatter(const int *__restrict__ src, const int *__restrict__ dst, int64_t m, int n, unsigned flags, int vbits,
                 BucketPlan *plan, int *status, unsigned *__restrict__ packed)
{
    extern __shared__ __align__(16) unsigned char bk_smem[];
    auto &sh = *reinterpret_cast<BucketShared *>(bk_smem);
    const bool sym = flags & GBFS_SYMMETRIZE, noself = flags & GBFS_DROP_SELF_LOOPS;
    const int t = (int)threadIdx.x;
    constexpr int64_t TILE = BK_SBLOCK * BK_EDGES;
    for (int64_t base = (int64_t)blockIdx.x * TILE; base < m; base += (int64_t)gridDim.x * TILE) {
        for (int b = t; b < BK_BUCKETS; b += BK_SBLOCK) sh.run[b].x = 0;
        int u[BK_EDGES], v[BK_EDGES];
#pragma unroll
        for (int q = 0; q < BK_EDGES; q++) load_edge(src, dst, base + q * BK_SBLOCK + t, m, n, noself, status, u[q], v[q]);
        // the next tile's edges on their way to L2
        const int64_t ahead = base + (int64_t)gridDim.x * TILE + 32 * (int64_t)t;
        if (32 * t < TILE && ahead < m) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(src + ahead));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(dst + ahead));
        }
        __syncthreads();
        unsigned rank[BK_EDGES];  // within the tile's runs: of (u -> v), and << 16 of (v -> u)
#pragma unroll
        for (int q = 0; q < BK_EDGES; q++) {
            rank[q] = 0;
            if (u[q] < 0) continue;
            rank[q] = (unsigned)atomicAdd(&sh.run[u[q] >> BK_LOG].x, 1);
            if (sym) rank[q] |= (unsigned)atomicAdd(&sh.run[v[q] >> BK_LOG].x, 1) << 16;
        }
        __syncthreads();
        int c[BK_PER], sum = 0;
#pragma unroll
        for (int k = 0; k < BK_PER; k++) {
            c[k] = sh.run[k * BK_SBLOCK + t].x;
            sum += c[k];
        }
        int total;
        int at = block_excl_scan(sum, sh.warp, &total);
#pragma unroll
        for (int k = 0; k < BK_PER; k++) {
            sh.run[k * BK_SBLOCK + t] = make_int2(at, c[k] ? atomicAdd(&plan->cursor[k * BK_SBLOCK + t], c[k]) : 0);
            at += c[k];
        }
        __syncthreads();
        auto put = [&](int row, int colv, unsigned r) {
            const int2 run = sh.run[row >> BK_LOG];
            sh.entry[run.x + r] =
                make_uint2((unsigned)(row & ((1 << BK_LOG) - 1)) << vbits | (unsigned)colv, (unsigned)run.y + r);
        };
#pragma unroll
        for (int q = 0; q < BK_EDGES; q++) {
            if (u[q] < 0) continue;
            put(u[q], v[q], rank[q] & 0xffffu);
            if (sym) put(v[q], u[q], rank[q] >> 16);
        }
        __syncthreads();
        for (int j = t; j < total; j += BK_SBLOCK) {
            const uint2 x = sh.entry[j];
            packed[x.y] = x.x;
        }
        __syncthreads();
    }
}

// agg_atomic_add on shared memory, where only a row that several lanes hit at
// once is worth a group (one atomic instead of a conflict per lane): the lanes
// that share lane 0's key, if they are half of them.
__device__ __forceinline__ int shared_rank_add(int *arr, int key)
{
    const unsigned same = __ballot_sync(FULL, key == __shfl_sync(FULL, key, 0));
    const bool grouped = __popc(same) >= 16;
    const bool mine = grouped && (same >> lane_id() & 1u);
    int old = 0;
    if (key >= 0 && (!mine || lane_id() == 0)) old = atomicAdd(arr + key, mine ? __popc(same) : 1);
    if (!grouped) return old;
    const int base = __shfl_sync(FULL, old, 0);
    return mine ? base + __popc(same & lanemask_lt()) : old;
}

// One CTA per bucket: row offsets, and the words replaced by the columns in
// their rows (in no particular order within a row), put together in shared
// memory where the bucket fits there (a scattered global store costs a cycle per
// lane), else in the spare buffer.
__global__ void __launch_bounds__(BK_BLOCK, 1)
k_bucket_rows(const BucketPlan *__restrict__ plan, unsigned *packed, int vbits, int n, int *row, int *spare)
{
    extern __shared__ int s_stage[];  // BK_STAGE columns
    __shared__ int s_cnt[1 << BK_LOG];
    __shared__ int s_warp[33];
    static_assert(BK_BLOCK == 1 << BK_LOG, "a thread per row");
    const int t = (int)threadIdx.x, b = plan->order[blockIdx.x];
    const int s = plan->start[b], e = plan->start[b + 1];
    const unsigned mask = (1u << vbits) - 1u;
    s_cnt[t] = 0;
    __syncthreads();
    auto load = [&](int i) { return packed[i]; };
    walk_range<BK_BLOCK, BK_ILP>(s, e, t, load,
                                 [&](unsigned w, bool in) { shared_rank_add(s_cnt, in ? (int)(w >> vbits) : -1); });
    __syncthreads();
    const int c = s_cnt[t];
    int total;
    const int off = block_excl_scan(c, s_warp, &total);
    const int v = (b << BK_LOG) + t;
    if (v < n) row[v] = s + off;
    if (v == n - 1) row[n] = s + off + c;
    s_cnt[t] = off;
    __syncthreads();
    const bool staged = e - s <= BK_STAGE;
    int *const over = spare + plan->over_at[b];
    walk_range<BK_BLOCK, BK_ILP>(s, e, t, load, [&](unsigned w, bool in) {
        const int pos = shared_rank_add(s_cnt, in ? (int)(w >> vbits) : -1);
        if (!in) return;
        if (staged) s_stage[pos] = (int)(w & mask);
        else over[pos] = (int)(w & mask);
    });
    __syncthreads();  // every word has been read
    for (int i = t; i < e - s; i += BK_BLOCK) packed[s + i] = (unsigned)(staged ? s_stage[i] : over[i]);
}

struct BinLists {
    int *list[BIN_CLASSES];
};
// What k_bin counts: rows per class, and the long rows' entries, chunks of
// MED_MAX, and longest row.
struct BinCounts {
    unsigned long long long_entries;
    unsigned rows[BIN_CLASSES];
    unsigned chunks;
    int longest;
};

// Rows longer than 32 go to a list by length.  A CTA ranks its rows with
// shared counters and takes its places with one global atomic per class
// (RMAT-22: 96 us with a block scan per class, 30 us so).
template <typename RT>
__global__ void k_bin(const RT *__restrict__ row, int n, BinLists lists, BinCounts *cnt)
{
    __shared__ unsigned s_cnt[BIN_CLASSES], s_base[BIN_CLASSES], s_chunks;
    __shared__ unsigned long long s_entries;
    __shared__ int s_longest;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x < BIN_CLASSES) s_cnt[threadIdx.x] = 0;
        if (threadIdx.x == 0) {
            s_chunks = 0;
            s_entries = 0;
            s_longest = 0;
        }
        __syncthreads();
        const int64_t r = base + threadIdx.x;
        const int d = r < n ? (int)(row[r + 1] - row[r]) : 0;
        const int cls = d <= 32       ? -1
                        : d <= W4_MAX  ? BIN_W4
                        : d <= W16_MAX ? BIN_W16
                        : d <= 1024    ? BIN_1K
                        : d <= 2048    ? BIN_2K
                        : d <= MED_MAX ? BIN_4K
                                       : BIN_LONG;
        unsigned off = 0;
        if (cls >= 0) off = atomicAdd(&s_cnt[cls], 1u);
        if (cls == BIN_LONG) {
            atomicAdd(&s_chunks, (unsigned)((d + MED_MAX - 1) / MED_MAX));
            atomicAdd(&s_entries, (unsigned long long)d);
            atomicMax(&s_longest, d);
        }
        __syncthreads();
        if (threadIdx.x < BIN_CLASSES)
            s_base[threadIdx.x] = s_cnt[threadIdx.x] ? atomicAdd(&cnt->rows[threadIdx.x], s_cnt[threadIdx.x]) : 0u;
        if (threadIdx.x == BIN_CLASSES && s_chunks) {
            atomicAdd(&cnt->chunks, s_chunks);
            atomicAdd(&cnt->long_entries, s_entries);
            atomicMax(&cnt->longest, s_longest);
        }
        __syncthreads();
        if (cls >= 0) {
            int *list = lists.list[0];
#pragma unroll
            for (int c = 1; c < BIN_CLASSES; c++)
                if (cls == c) list = lists.list[c];
            list[s_base[cls] + off] = (int)r;
        }
    }
}

__device__ __forceinline__ int warp_bitonic_sort(int x)
{
    const unsigned lane = lane_id();
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            int y = __shfl_xor_sync(FULL, x, j);
            bool up = (lane & k) == 0;
            bool lower = (lane & j) == 0;
            x = (lower == up) ? min(x, y) : max(x, y);
        }
    }
    return x;
}

// Sorts 8 values ascending (Batcher's odd-even merge network, 19 exchanges).
__device__ __forceinline__ void sort8(int (&v)[8])
{
    auto cx = [&](int a, int b) {
        const int lo = min(v[a], v[b]), hi = max(v[a], v[b]);
        v[a] = lo;
        v[b] = hi;
    };
    cx(0, 1); cx(2, 3); cx(4, 5); cx(6, 7);
    cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7);
    cx(1, 2); cx(5, 6);
    cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7);
    cx(2, 4); cx(3, 5);
    cx(1, 2); cx(3, 4); cx(5, 6);
}

// Rows of length <= 32: sort in registers, pack distinct values.  A warp loads
// the offsets of 32 consecutive rows at once.  Rows of up to 8 entries are
// sorted by a lane each, all 32 at once (a grid of 16 M vertices: 1.93 ms with
// a warp per row, 0.13 ms so), rows of up to 16 by half a warp, two at a time,
// the others by the warp, one after another.
template <typename RT>
__global__ void k_sort_small(const RT *__restrict__ row, int n, int *tmp, int dedup, int *ucnt)
{
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned lane = lane_id();
    for (int64_t r0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; r0 < n; r0 += warps * 32) {
        RT bl = 0;
        int dl = 33;  // rows past n are skipped as long ones
        if (r0 + lane < n) {
            bl = row[r0 + lane];
            dl = (int)(row[r0 + lane + 1] - bl);
        }
        if (dl <= 8) {
            int v[8], k = 0;
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = e < dl ? tmp[bl + e] : INT_MAX;
            sort8(v);
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (e < dl && (!dedup || e == 0 || v[e] != v[e - 1])) tmp[bl + k++] = v[e];
            ucnt[r0 + lane] = k;
        }
        __syncwarp();
        // half a warp per row: the first two rows left, and so on
        unsigned left = __ballot_sync(FULL, dl > 8 && dl <= 16);
        while (left) {
            const int j0 = __ffs(left) - 1;
            left &= left - 1u;
            const int j1 = left ? __ffs(left) - 1 : j0;
            const bool two = left != 0;
            if (two) left &= left - 1u;
            const unsigned h = lane & 15u;
            const int j = lane < 16 ? j0 : j1;
            const RT b = __shfl_sync(FULL, bl, j);
            const int d = __shfl_sync(FULL, dl, j);
            const bool on = lane < 16 || two;
            int x = on && (int)h < d ? tmp[b + h] : INT_MAX;
#pragma unroll
            for (int k = 2; k <= 16; k <<= 1)
#pragma unroll
                for (int i = k >> 1; i > 0; i >>= 1) {
                    const int y = __shfl_xor_sync(FULL, x, i);
                    x = ((h & i) == 0) == ((h & k) == 0) ? min(x, y) : max(x, y);
                }
            const int prev = __shfl_up_sync(FULL, x, 1);
            const bool keep = on && (int)h < d && (!dedup || h == 0 || x != prev);
            const unsigned mask = __ballot_sync(FULL, keep) >> (lane & 16u) & 0xffffu;
            if (keep) tmp[b + __popc(mask & ((1u << h) - 1u))] = x;
            if (on && h == 0) ucnt[r0 + j] = __popc(mask);
        }
        left = __ballot_sync(FULL, dl > 16 && dl <= 32);
        while (left) {
            const int j = __ffs(left) - 1;
            left &= left - 1u;
            const RT b = __shfl_sync(FULL, bl, j);
            const int d = __shfl_sync(FULL, dl, j);
            int x = (int)lane < d ? tmp[b + lane] : INT_MAX;
            x = warp_bitonic_sort(x);
            const int prev = __shfl_up_sync(FULL, x, 1);
            const bool keep = (int)lane < d && (!dedup || lane == 0 || x != prev);
            const unsigned mask = __ballot_sync(FULL, keep);
            if (keep) tmp[b + __popc(mask & lanemask_lt())] = x;
            if (lane == 0) ucnt[r0 + j] = __popc(mask);
        }
    }
}

// Bitonic sort of 32*E values held E per lane (element i = lane i%32,
// register i/32), ascending.  Compare-exchange distances below 32 go
// through shuffles, larger ones between a lane's own registers; all loops
// unroll, so the registers stay registers.
template <int E>
__device__ __forceinline__ void warp_bitonic_sort_regs(int (&v)[E])
{
    const int lane = (int)lane_id();
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const int r2 = r ^ (j >> 5);
                    if (r2 > r) {
                        const bool up = ((r * 32 + lane) & k) == 0;
                        const int a = v[r], c = v[r2];
                        if ((a > c) == up) {
                            v[r] = c;
                            v[r2] = a;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const int y = __shfl_xor_sync(FULL, v[r], j);
                    const bool up = ((r * 32 + lane) & k) == 0;
                    const bool lower = (lane & j) == 0;
                    v[r] = (lower == up) ? min(v[r], y) : max(v[r], y);
                }
            }
        }
    }
}

// One warp per listed row of length 33..32*E: sort in registers, pack the
// distinct values (dedup) or all of them back in place, record the count.
template <int E, typename RT>
__global__ void k_sort_warp(const RT *__restrict__ row, const int *__restrict__ list, const unsigned *cnt,
                            int *tmp, int dedup, int *ucnt)
{
    const int count = (int)*cnt;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = (int)lane_id();
    for (int64_t li = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; li < count; li += warps) {
        const int r = list[li];
        const RT b = row[r];
        const int d = (int)(row[r + 1] - b);
        int v[E];
#pragma unroll
        for (int k = 0; k < E; k++) {
            const int i = k * 32 + lane;
            v[k] = i < d ? tmp[b + i] : INT_MAX;
        }
        warp_bitonic_sort_regs<E>(v);
        int base = 0;
#pragma unroll
        for (int k = 0; k < E; k++) {
            const int i = k * 32 + lane;
            int prev = __shfl_up_sync(FULL, v[k], 1);
            if (k > 0) {
                const int last = __shfl_sync(FULL, v[k - 1], 31);
                if (lane == 0) prev = last;
            }
            const bool keep = i < d && (!dedup || i == 0 || v[k] != prev);
            const unsigned mk = __ballot_sync(FULL, keep);
            if (keep) tmp[b + base + __popc(mk & lanemask_lt())] = v[k];
            base += __popc(mk);
        }
        if (lane == 0) ucnt[r] = base;
    }
}

// Sorts the CTA's T * SB_E values ascending: afterwards thread t holds values
// t * SB_E .. t * SB_E + 7.  A bitonic network in which exchanges between a
// thread's own values and between lanes of a warp stay in registers (68 of
// the 78 steps of 4096 values) and the others go through shared memory (buf:
// two buffers of T * SB_E values, so a step needs one barrier).  The network
// with every step in shared memory took 3.6 ms for the rows of 513 to 4096
// entries of RMAT-22 (50 M entries); this takes 0.6 ms.
template <int T>
__device__ __forceinline__ void block_bitonic_sort(int (&v)[SB_E], int *buf)
{
    const int t = (int)threadIdx.x;
    int4 *b4 = reinterpret_cast<int4 *>(buf);
    int flip = 0;
#pragma unroll
    for (int k = 2; k <= T * SB_E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j < SB_E) {
#pragma unroll
                for (int e = 0; e < SB_E; e++) {
                    const int p = e ^ j;
                    if (p > e) {
                        const bool up = ((t * SB_E + e) & k) == 0;
                        const int lo = min(v[e], v[p]), hi = max(v[e], v[p]);
                        v[e] = up ? lo : hi;
                        v[p] = up ? hi : lo;
                    }
                }
            } else {
                const bool keep_min = (((t * SB_E) & k) == 0) == (((t * SB_E) & j) == 0);
                int y[SB_E];
                if (j < 32 * SB_E) {
#pragma unroll
                    for (int e = 0; e < SB_E; e++) y[e] = __shfl_xor_sync(FULL, v[e], j / SB_E);
                } else {
                    int4 *s = b4 + flip * (T * SB_E / 4);
                    flip ^= 1;
                    // the two halves of a thread's values apart: consecutive
                    // threads' 16-byte accesses are then consecutive
                    s[t] = make_int4(v[0], v[1], v[2], v[3]);
                    s[T + t] = make_int4(v[4], v[5], v[6], v[7]);
                    __syncthreads();
                    const int4 a = s[t ^ (j / SB_E)], c = s[T + (t ^ (j / SB_E))];
                    y[0] = a.x; y[1] = a.y; y[2] = a.z; y[3] = a.w;
                    y[4] = c.x; y[5] = c.y; y[6] = c.z; y[7] = c.w;
                }
#pragma unroll
                for (int e = 0; e < SB_E; e++) v[e] = keep_min ? min(v[e], y[e]) : max(v[e], y[e]);
            }
        }
    }
    __syncthreads();
}

// Packs the CTA's sorted values (thread t: values t * SB_E ..., the first d of
// them real) into out: all of them, or (dedup) those that differ from their
// predecessor; `before`: the value before the first (INT_MIN: none).  Returns
// the count.  buf: T * SB_E values of shared memory.
template <int T>
__device__ __forceinline__ int block_pack(const int (&v)[SB_E], int d, bool dedup, int before, int *out, int *buf,
                                          int *s_warp)
{
    __shared__ int s_last[T / 32];
    const int t = (int)threadIdx.x;
    if (lane_id() == 31) s_last[t >> 5] = v[SB_E - 1];
    int prev = __shfl_up_sync(FULL, v[SB_E - 1], 1);
    __syncthreads();
    if (lane_id() == 0) prev = t == 0 ? before : s_last[(t >> 5) - 1];
    unsigned keep = 0;
#pragma unroll
    for (int e = 0; e < SB_E; e++) {
        const int p = e ? v[e - 1] : prev;
        if (t * SB_E + e < d && (!dedup || v[e] != p)) keep |= 1u << e;
    }
    int total;
    int off = block_excl_scan(__popc(keep), s_warp, &total);
#pragma unroll
    for (int e = 0; e < SB_E; e++)
        if (keep >> e & 1u) buf[off++] = v[e];
    __syncthreads();
    if (out)
        for (int i = t; i < total; i += T) out[i] = buf[i];
    __syncthreads();
    return total;
}

// One CTA of T threads per listed row of up to T * SB_E entries: sort in
// registers, pack in place, record the count.
template <int T, typename RT>
__global__ void __launch_bounds__(T) k_sort_block(const RT *__restrict__ row, const int *__restrict__ list,
                                                  const unsigned *cnt, int *tmp, int dedup, int *ucnt)
{
    __shared__ __align__(16) int s[2 * T * SB_E];
    __shared__ int s_warp[33];
    const int count = (int)*cnt;
    for (int li = blockIdx.x; li < count; li += gridDim.x) {
        const int r = list[li];
        const RT b = row[r];
        const int d = (int)(row[r + 1] - b);
        int v[SB_E];
#pragma unroll
        for (int e = 0; e < SB_E; e++) {
            const int i = e * T + (int)threadIdx.x;  // any order will do before the sort
            v[e] = i < d ? tmp[b + i] : INT_MAX;
        }
        block_bitonic_sort<T>(v, s);
        const int total = block_pack<T>(v, d, dedup, INT_MIN, tmp + b, s, s_warp);
        if (threadIdx.x == 0) ucnt[r] = total;
    }
}

// ---- rows longer than MED_MAX ----
// Distinct values of rows over not too many vertices: a bitmap of the vertices
// in shared memory, of which each CTA of a cluster holds a range.  All CTAs read
// the row and set their range's bits, count them, and after the cluster barrier
// (every entry has been read, and every CTA's count is known to the others)
// write their range's values over the row, in ascending order.  A row costs two
// reads of the bitmap and no comparisons.  What bounds it: the smem atomics of a
// row's entries, and a handful of barriers per row (two CTAs per SM overlap
// them; one CTA with twice the threads and range was 1 % slower).  Builds with
// the long rows sorted in chunks and merged, and so: RMAT-22 6.95 and 6.30 ms
// (their kernels 0.98 and 0.6), RMAT-21 3.89 and 3.33, RMAT-20 2.52 and 2.07,
// 4,096 vertices of 4,096 neighbours 4.75 and 3.77.  More CTAs per row mean more
// readers of its entries and more of the bitmap per entry: RMAT-23 with five CTAs
// of twice the range 16.7 and 16.6 ms, so larger graphs keep the chunks.  Rows of
// 2,049 to 4,096 entries pay off where one or two CTAs hold the bitmap (RMAT-20
// 2.07 and 2.04 ms, RMAT-19 1.50 and 1.46; RMAT-22 6.45 and 7.48).

constexpr int BMR_THREADS = 512;
constexpr int BMR_WORDS = 53;    // words of the bitmap per thread, at most
constexpr int BMR_CTAS = 5;      // CTAs of the largest cluster (4.3 M vertices)
constexpr int BMR_CTAS_4K = 2;   // and where rows of 2,049 to 4,096 entries take part
constexpr int BMR_ILP = 8;       // a thread's entries in flight
constexpr int BMR_CLUSTERS = 16; // clusters per one that the SMs hold (long rows differ much:
                                 // RMAT-22 6.45 ms with 2, 6.37 with 16)

// Words per thread (odd: the lanes' pieces start on different banks) and CTAs per
// row for n vertices.
struct BitmapShape {
    int words, ctas;
    explicit BitmapShape(int64_t n)
    {
        const int64_t all = (n + 32 * BMR_THREADS - 1) / (32 * BMR_THREADS);
        ctas = (int)((all + BMR_WORDS - 1) / BMR_WORDS);
        words = (int)((all + ctas - 1) / ctas) | 1;
    }
    size_t smem() const { return sizeof(unsigned) * BMR_THREADS * (size_t)words; }
};

template <typename RT>
__global__ void __launch_bounds__(BMR_THREADS)
k_long_rows(const RT *__restrict__ row, const int *__restrict__ list, const unsigned *cnt, int words, int *tmp,
            int *ucnt)
{
    extern __shared__ __align__(16) unsigned s_bits[];
    __shared__ int s_warp[33];
    __shared__ int s_count[2][BMR_CTAS];  // each CTA's, by the parity of the cluster's row
    const int t = (int)threadIdx.x;
    const unsigned rank = cluster_rank(), ctas = cluster_size();
    const unsigned range = 32u * BMR_THREADS * (unsigned)words, v0 = rank * range;
    unsigned *const mine = s_bits + t * words;
    for (int k = 0; k < words; k++) mine[k] = 0;
    cluster_barrier();  // the bitmaps are clear, and every CTA has started: the first row's counts may go out
    const int count = (int)*cnt, step = (int)(gridDim.x / ctas);
    int par = 0, li = (int)(blockIdx.x / ctas);
    int r = 0, rn = li < count ? list[li] : 0;  // the row, and the next one
    RT b = 0, bn = row[rn], en = row[rn + 1];
    for (; li < count; li += step, par ^= 1) {
        r = rn;
        b = bn;
        const int d = (int)(en - b);
        int *const at = tmp + b;
        if (li + step < count) rn = list[li + step];
        for (unsigned i0 = (unsigned)t; i0 < (unsigned)d; i0 += BMR_ILP * BMR_THREADS) {
            unsigned u[BMR_ILP];
#pragma unroll
            for (int q = 0; q < BMR_ILP; q++) {
                const unsigned i = i0 + (unsigned)(q * BMR_THREADS);
                u[q] = i < (unsigned)d ? (unsigned)at[i] - v0 : range;
            }
#pragma unroll
            for (int q = 0; q < BMR_ILP; q++)
                if (u[q] < range) atomicOr(&s_bits[u[q] >> 5], 1u << (u[q] & 31));
        }
        bn = row[rn];
        en = row[rn + 1];
        __syncthreads();
        unsigned set[2] = {0, 0};  // this thread's words with set bits
        int c = 0, total;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll 8
            for (int k = 32 * h; k < min(words, 32 * h + 32); k++) {
                const unsigned w = mine[k];
                c += __popc(w);
                if (w) set[h] |= 1u << (k - 32 * h);
            }
        int o = block_excl_scan(c, s_warp, &total);
        if (t < (int)ctas)
            remote_store_u32(map_rank(smem_addr(&s_count[par][rank]), (unsigned)t), (unsigned)total);
        cluster_barrier();
        int all = 0;
        for (unsigned k = 0; k < ctas; k++) {
            if (k == rank) o += all;
            all += s_count[par][k];
        }
        if (rank == 0 && t == 0) ucnt[r] = all;
#pragma unroll
        for (int h = 0; h < 2; h++)
            while (set[h]) {
                const int k = 32 * h + __ffs(set[h]) - 1;
                set[h] &= set[h] - 1;
                unsigned w = mine[k];
                mine[k] = 0;
                const int v = (int)(v0 + 32u * (unsigned)(t * words + k));
                while (w) {
                    at[o++] = v + __ffs(w) - 1;
                    w &= w - 1;
                }
            }
        __syncthreads();  // the bitmap is clear
    }
}

// Copies the packed long rows, each by up to eight CTAs.
constexpr int CPL_THREADS = 512, CPL_PER = 8;

template <typename RT>
__global__ void __launch_bounds__(CPL_THREADS)
k_compact_long(const RT *__restrict__ row, const RT *__restrict__ row2, const int *__restrict__ list,
               const int *__restrict__ tmp, int *col)
{
    const int r = list[blockIdx.x];
    const int *const from = tmp + row[r];
    int *const to = col + row2[r];
    const int c = (int)(row2[r + 1] - row2[r]);
    for (int64_t i0 = (int64_t)blockIdx.y * (CPL_THREADS * CPL_PER); i0 < c;
         i0 += (int64_t)gridDim.y * (CPL_THREADS * CPL_PER)) {
        int x[CPL_PER];
#pragma unroll
        for (int q = 0; q < CPL_PER; q++) {
            const int64_t i = i0 + q * CPL_THREADS + threadIdx.x;
            x[q] = i < c ? from[i] : 0;
        }
#pragma unroll
        for (int q = 0; q < CPL_PER; q++) {
            const int64_t i = i0 + q * CPL_THREADS + threadIdx.x;
            if (i < c) to[i] = x[q];
        }
    }
}

// Other long rows:
// A long row is sorted in chunks of MED_MAX, all chunks of all such rows at
// once, and its chunks are merged pairwise, one tile of MED_MAX outputs per
// CTA.  RMAT-22 has 1,794 long rows of 25.5 M entries, the longest 320 K: a
// radix sort by one CTA per row took 3.5 ms, with that row its tail; chunks
// and seven merge passes take 0.8 ms.

// The j-th chunk of a row, and where in tmp2 the row's entries have their
// second place.
struct Chunk {
    long long base2;
    int row, j;
};
struct ChunkNext {
    unsigned long long entries;
    unsigned chunks, pad;
};

// The chunks of every listed row; a row's are consecutive.
template <typename RT>
__global__ void k_chunks(const RT *__restrict__ row, const int *__restrict__ list, const unsigned *cnt, Chunk *chunks,
                         ChunkNext *next)
{
    const int count = (int)*cnt;
    for (int li = blockIdx.x * blockDim.x + threadIdx.x; li < count; li += gridDim.x * blockDim.x) {
        const int r = list[li];
        const int d = (int)(row[r + 1] - row[r]);
        const int nc = (d + MED_MAX - 1) / MED_MAX;
        const unsigned at = atomicAdd(&next->chunks, (unsigned)nc);
        const long long base2 = (long long)atomicAdd(&next->entries, (unsigned long long)d);
        for (int j = 0; j < nc; j++) chunks[at + j] = Chunk{base2, r, j};
    }
}

// Merge passes a row of d entries needs.
__host__ __device__ inline int merge_passes(int d)
{
    int p = 0;
    while (((int64_t)MED_MAX << p) < d) p++;
    return p;
}

// Sorts every chunk, into tmp2 where the row's number of merge passes is odd
// (so that its last pass ends in tmp).
template <typename RT>
__global__ void __launch_bounds__(MED_THREADS)
k_sort_chunks(const RT *__restrict__ row, const Chunk *__restrict__ chunks, int nchunks, int *tmp, int *tmp2)
{
    __shared__ __align__(16) int s[2 * MED_MAX];
    __shared__ int s_warp[33];
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const Chunk ck = chunks[c];
        const RT rb = row[ck.row];
        const int len = (int)(row[ck.row + 1] - rb), at = ck.j * MED_MAX;
        const int d = min(MED_MAX, len - at);
        int *from = tmp + rb + at;
        int v[SB_E];
#pragma unroll
        for (int e = 0; e < SB_E; e++) {
            const int i = e * MED_THREADS + (int)threadIdx.x;
            v[e] = i < d ? from[i] : INT_MAX;
        }
        block_bitonic_sort<MED_THREADS>(v, s);
        block_pack<MED_THREADS>(v, d, false, INT_MIN, merge_passes(len) & 1 ? tmp2 + ck.base2 + at : from, s, s_warp);
    }
}

// How many of the first o merged values of ascending A (na) and B (nb) come
// from A (equal values: A first).
__device__ __forceinline__ int merge_split(const int *A, int na, const int *B, int nb, int o)
{
    int lo = max(0, o - nb), hi = min(o, na);
    while (lo < hi) {
        const int i = (lo + hi) >> 1;
        if (A[i] <= B[o - 1 - i]) lo = i + 1; else hi = i;
    }
    return lo;
}

// Pass p: runs of MED_MAX << p are merged in pairs.  A chunk's CTA makes the
// outputs in its place, from one of the row's two places to the other.
template <typename RT>
__global__ void __launch_bounds__(MED_THREADS)
k_merge(const RT *__restrict__ row, const Chunk *__restrict__ chunks, int nchunks, int *tmp, int *tmp2, int p)
{
    __shared__ int s[MED_MAX];
    __shared__ int s_split[2];
    const int t = (int)threadIdx.x;
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const Chunk ck = chunks[c];
        const RT rb = row[ck.row];
        const int d = (int)(row[ck.row + 1] - rb);
        const int left = merge_passes(d) - p;  // passes from here on
        if (left <= 0) continue;               // this row is done
        int *one = tmp + rb, *two = tmp2 + ck.base2;
        const int *from = left & 1 ? two : one;
        int *to = left & 1 ? one : two;
        const int64_t w = (int64_t)MED_MAX << p;
        const int a0 = (ck.j >> (p + 1)) * (int)min(2 * w, (int64_t)INT_MAX);
        const int b0 = (int)min((int64_t)d, a0 + w), b1 = (int)min((int64_t)d, a0 + 2 * w);
        const int o0 = ck.j * MED_MAX - a0, o1 = min(o0 + MED_MAX, b1 - a0);
        const int *A = from + a0, *B = from + b0;
        const int na = b0 - a0, nb = b1 - b0;
        if (t < 64 && (t & 31) == 0) s_split[t >> 5] = merge_split(A, na, B, nb, t ? o1 : o0);
        __syncthreads();
        const int i0 = s_split[0], i1 = s_split[1];
        const int ta = i1 - i0, tb = (o1 - o0) - ta;
        for (int i = t; i < ta; i += MED_THREADS) s[i] = A[i0 + i];
        for (int i = t; i < tb; i += MED_THREADS) s[ta + i] = B[o0 - i0 + i];
        __syncthreads();
        int v[SB_E];
        const int o = min(t * SB_E, ta + tb);
        int ia = merge_split(s, ta, s + ta, tb, o), ib = o - ia;
#pragma unroll
        for (int e = 0; e < SB_E; e++) {
            const bool a = ia < ta && (ib >= tb || s[ia] <= s[ta + ib]);
            v[e] = INT_MAX;
            if (a) v[e] = s[ia++];
            else if (ib < tb) v[e] = s[ta + ib++];
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < SB_E; e++)
            if (o + e < ta + tb) s[o + e] = v[e];
        __syncthreads();
        for (int i = t; i < ta + tb; i += MED_THREADS) to[ck.j * MED_MAX + i] = s[i];
        __syncthreads();
    }
}

// Distinct values of every merged chunk (a value equal to the one before the
// chunk is not counted), added up per row in ucnt (zeroed by the caller).
template <typename RT>
__global__ void __launch_bounds__(MED_THREADS)
k_chunk_unique(const RT *__restrict__ row, const Chunk *__restrict__ chunks, int nchunks, const int *__restrict__ tmp,
               int *ccnt, int *ucnt)
{
    __shared__ int s_red[32];
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const Chunk ck = chunks[c];
        const RT b = row[ck.row] + (RT)ck.j * MED_MAX;
        const int d = (int)min((RT)MED_MAX, row[ck.row + 1] - b);
        const int *from = tmp + b;
        int mine = 0;
        for (int i = threadIdx.x; i < d; i += MED_THREADS) mine += (i == 0 && ck.j == 0) || from[i] != from[i - 1];
        const int total = block_sum(mine, s_red);
        if (threadIdx.x == 0) {
            ccnt[c] = total;
            atomicAdd(&ucnt[ck.row], total);
        }
    }
}

// The distinct values of every merged chunk into its row of col.
template <typename RT>
__global__ void __launch_bounds__(MED_THREADS)
k_compact_chunks(const RT *__restrict__ row, const RT *__restrict__ row2, const Chunk *__restrict__ chunks,
                 int nchunks, const int *__restrict__ ccnt, const int *__restrict__ tmp, int *col)
{
    __shared__ int s[MED_MAX];
    __shared__ int s_warp[33];
    __shared__ int s_red[32], s_rel;
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const Chunk ck = chunks[c];
        int rel = 0;  // distinct values in the row's earlier chunks
        for (int i = threadIdx.x; i < ck.j; i += MED_THREADS) rel += ccnt[c - ck.j + i];
        rel = block_sum(rel, s_red);
        if (threadIdx.x == 0) s_rel = rel;
        const RT b = row[ck.row] + (RT)ck.j * MED_MAX;
        const int d = (int)min((RT)MED_MAX, row[ck.row + 1] - b);
        for (int i = threadIdx.x; i < d; i += MED_THREADS) s[i] = tmp[b + i];
        __syncthreads();
        int v[SB_E];
#pragma unroll
        for (int e = 0; e < SB_E; e++) {
            const int i = (int)threadIdx.x * SB_E + e;
            v[e] = i < d ? s[i] : INT_MAX;
        }
        int *out = col + row2[ck.row] + s_rel;
        __syncthreads();
        block_pack<MED_THREADS>(v, d, true, ck.j ? tmp[b - 1] : INT_MIN, out, s, s_warp);
    }
}

// Copy the packed distinct prefix of each row.  A warp loads the offsets of 32
// consecutive rows at once; rows of up to 64 entries are copied as one
// concatenated range (a lane finds its entry's row with shuffles), longer ones
// one after another (all rows one after another: 0.50 ms for a grid of 16 M
// vertices, 0.17 so).
template <typename RT>
__global__ void k_compact(const RT *__restrict__ row, const RT *__restrict__ row2, int n,
                          const int *__restrict__ tmp, int *col)
{
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = (int)lane_id();
    for (int64_t r0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; r0 < n; r0 += warps * 32) {
        const int64_t r = r0 + lane;
        RT b = 0, o = 0;
        int c = 0;
        // rows longer than MED_MAX before deduplication: k_compact_chunks
        if (r < n && row[r + 1] - row[r] <= MED_MAX) {
            b = row[r];
            o = row2[r];
            c = (int)(row2[r + 1] - o);
        }
        const int cs = c <= 64 ? c : 0;
        const int incl = warp_incl_scan(cs), excl = incl - cs;
        const int T = __shfl_sync(FULL, incl, 31);
        for (int e0 = 0; e0 < T; e0 += 64) {
            int x[2];
            RT at[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int e = e0 + q * 32 + lane, ee = min(e, T - 1);
                int j = 0;  // the last row that starts at or before entry ee
#pragma unroll
                for (int s = 16; s > 0; s >>= 1)
                    if (__shfl_sync(FULL, excl, j + s) <= ee) j += s;
                const int k = ee - __shfl_sync(FULL, excl, j);
                const RT from = __shfl_sync(FULL, b, j) + k;
                at[q] = __shfl_sync(FULL, o, j) + k;
                x[q] = e < T ? tmp[from] : 0;
            }
#pragma unroll
            for (int q = 0; q < 2; q++)
                if (e0 + q * 32 + lane < T) col[at[q]] = x[q];
        }
        unsigned left = __ballot_sync(FULL, c > 64);
        while (left) {
            const int j = __ffs(left) - 1;
            left &= left - 1u;
            const RT bj = __shfl_sync(FULL, b, j), oj = __shfl_sync(FULL, o, j);
            const int cj = __shfl_sync(FULL, c, j);
#pragma unroll 4
            for (int i = lane; i < cj; i += 32) col[oj + i] = tmp[bj + i];
        }
    }
}

// SMALL: with the costs of the parts that the one-cluster search deals in.
template <bool SMALL, typename RT>
__global__ void k_finalize(const RT *__restrict__ row, int n, unsigned *zmask, int *maxdeg,
                           unsigned long long *nonisolated, unsigned *nover4, unsigned long long *part, int part_log)
{
    __shared__ unsigned long long s_red[32];
    __shared__ int s_max[32];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // non-isolated rows, and rows of more than four entries in the high half
    unsigned long long mine = 0, cost = 0;
    int mx = 0;
    const int W = (n + 31) >> 5;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < (int64_t)W * 32;
         base += stride) {
        int64_t v = base + lane_id();
        int d = v < n ? (int)(row[v + 1] - row[v]) : 0;
        unsigned z = __ballot_sync(FULL, d == 0);  // out-of-range bits count as zero-degree
        if (lane_id() == 0) zmask[v >> 5] = z;
        mine += (d > 0 ? 1ull : 0ull) + (d > 4 ? 1ull << 32 : 0ull);
        if (SMALL) cost += (unsigned long long)small_row_cost(d);
        mx = max(mx, d);
    }
    if (SMALL) {  // (the grid covers so small a graph in one go: a CTA's vertices are of one part)
        cost = block_sum(cost, s_red);
        if (threadIdx.x == 0 && cost) atomicAdd(part + ((blockIdx.x * blockDim.x) >> part_log), cost);
    }
    unsigned long long t = block_sum(mine, s_red);
    if (threadIdx.x == 0 && t) {
        atomicAdd(nonisolated, t & 0xffffffffull);
        if (t >> 32) atomicAdd(nover4, (unsigned)(t >> 32));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(FULL, mx, o));
    __syncthreads();
    if (lane_id() == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < (blockDim.x >> 5); w++) mx = max(mx, s_max[w]);
        atomicMax(maxdeg, mx);
    }
}

// Appends the rows with more than HEAVY_DEGREE entries to heavy, with one
// global atomic per CTA pass (one per warp, all on one counter, took 80 us on
// RMAT-22; this takes 22).
template <typename RT>
__global__ void k_heavy_list(const RT *__restrict__ row, int n, int *heavy, unsigned *cnt)
{
    __shared__ unsigned s_cnt, s_base;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += (int64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x == 0) s_cnt = 0;
        __syncthreads();
        const int64_t v = base + threadIdx.x;
        const bool h = v < n && row[v + 1] - row[v] > HEAVY_DEGREE;
        unsigned off = 0;
        if (h) off = atomicAdd(&s_cnt, 1u);
        __syncthreads();
        if (threadIdx.x == 0 && s_cnt) s_base = atomicAdd(cnt, s_cnt);
        __syncthreads();
        if (h) heavy[s_base + off] = (int)v;
        __syncthreads();
    }
}

template <typename RT>
__global__ void k_validate_csr(const RT *__restrict__ row, const int *__restrict__ col, int n,
                               int64_t m, int *status)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m || i < n; i += stride) {
        if (i < n && row[i + 1] < row[i]) atomicExch(status, DEV_BAD_ID);
        if (i < m && (unsigned)col[i] >= (unsigned)n) atomicExch(status, DEV_BAD_ID);
    }
}

// The first of 32 rows among which entry e's is, for a w with row[w] <= e: rows
// w + 1 to the one sought are empty or end before e.  Strides of 32, 32^2, ...
// rows as far as that is too few, then back down, 32 looks at once: a gap of g
// rows takes about 2 log32(g / 32) + 1 round trips (32 rows at a time, a gap of 5 M
// empty rows held one warp for 156,000).  The whole warp calls it.
template <typename RT>
__device__ __forceinline__ int skip_empty_rows(const RT *__restrict__ row, int n, int w, int64_t e)
{
    int64_t at = w, stride = 32;
    for (;; stride *= 32) {
        const int64_t x = at + (lane_id() + 1) * stride;
        const int k = __popc(__ballot_sync(FULL, x <= n && (int64_t)row[x <= n ? x : 0] <= e));
        at += k * stride;
        if (k < 32) break;
    }
    while (stride > 32) {
        stride /= 32;
        const int64_t x = at + (lane_id() + 1) * stride;
        at += stride * __popc(__ballot_sync(FULL, x <= n && (int64_t)row[x <= n ? x : 0] <= e));
    }
    return (int)at;
}

// Calls f(e, u, in) for the m entries e of the rows, u the entry's row: a warp
// takes EDGE_CHUNK consecutive entries at a time, 32 a step (in: the lane has
// one), so the work does not follow the rows' lengths.  All lanes call f; a step
// in which it returns true (to all of them) ends the warp's walk.
constexpr int EDGE_CHUNK = 1024;

template <typename RT, typename F>
__device__ __forceinline__ void for_edges(const RT *__restrict__ row, int n, int64_t m, F f)
{
    const int lane = (int)lane_id();
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = gw * EDGE_CHUNK; base < m; base += nw * EDGE_CHUNK) {
        int u = 0, hi = n;  // row[u] <= base < row[hi]
        while (hi - u > 1) {
            const int mid = u + (hi - u) / 2;
            if ((int64_t)row[mid] <= base) u = mid; else hi = mid;
        }
        const int64_t end = min(m, base + EDGE_CHUNK);
        for (int64_t e0 = base; e0 < end; e0 += 32) {
            const int64_t e = e0 + lane;
            const bool in = e < end;
            int mine = -1;
            for (int w = u;;) {  // 32 rows' ends at a time
                const int64_t at = (int64_t)w + 1 + lane, r = at <= n ? (int64_t)row[at] : INT64_MAX;
                int k = 0;  // of them at or before e
#pragma unroll
                for (int s = 16; s > 0; s >>= 1)
                    if (__shfl_sync(FULL, r, k + s - 1) <= e) k += s;
                if (__shfl_sync(FULL, r, k) <= e) ++k;
                const bool hit = mine < 0 && k < 32;
                if (hit) mine = w + k;
                const unsigned left = __ballot_sync(FULL, in && mine < 0);
                if (!left) break;
                w += 32;
                if (!__any_sync(FULL, in && hit)) w = skip_empty_rows(row, n, w, e0 + __ffs(left) - 1);
            }
            if (f(e, mine, in)) return;
            u = __shfl_sync(FULL, mine, (int)(min(end, e0 + 32) - e0) - 1);
        }
    }
}

// Whether sorted row v has an entry u.
template <typename RT>
__device__ __forceinline__ bool row_has(const RT *__restrict__ row, const int *__restrict__ col, int v, int u)
{
    const RT last = row[v + 1];
    RT lo = row[v], hi = last;
    while (lo < hi) {
        const RT mid = idx_mid(lo, hi);
        if (col[mid] < u) lo = mid + 1; else hi = mid;
    }
    return lo < last && col[lo] == u;
}

// Symmetry check on sorted rows: every (u,v) has (v,u).  A warp stops at its first
// entry without, which in a directed graph is soon enough (looking at the flag for
// what others have found costs more, as all warps' looks queue up in L2).
template <typename RT>
__global__ void k_check_sym(const RT *__restrict__ row, const int *__restrict__ col, int n, int64_t m, int *flags)
{
    for_edges(row, n, m, [&](int64_t e, int u, bool in) {
        const bool missing = in && !row_has(row, col, col[e], u);
        if (missing) flags[1] = 1;
        return __any_sync(FULL, missing) != 0;
    });
}

// The same with a thread per row (up to its first entry without), for graphs without rows of more than
// HEAVY_DEGREE entries, where finding each entry's row costs more than uneven
// rows: uniform random, 4 M vertices, 64 M entries: 1.76 ms against 2.33 by
// entries, a grid of 3000 x 3000 0.10 against 0.30; with a hub among the rows it
// would be the longest row's time (RMAT-20: 100 ms against 1.1).
template <typename RT>
__global__ void k_check_sym_rows(const RT *__restrict__ row, const int *__restrict__ col, int n, int *flags)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += stride) {
        const RT b = row[u], e = row[u + 1];
        bool missing = false;
        for (RT i = b; i < e && !missing; i++) missing = !row_has(row, col, col[i], (int)u);
        if (missing) {
            flags[1] = 1;
            return;
        }
    }
}

// Rows ascend where every descent of the column array is at a row's start:
// descents counted over all entries, less those at the rows' first ones.
template <typename RT>
__global__ void k_check_sorted(const RT *__restrict__ row, const int *__restrict__ col, int n, int64_t m,
                               unsigned long long *descents)
{
    __shared__ unsigned long long s_red[32];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long mine = 0;
    for (int64_t i = t + 1; i < m; i += stride) mine += col[i - 1] > col[i];
    for (int64_t u = t; u < n; u += stride) {
        const int64_t b = (int64_t)row[u];
        if (b > 0 && (int64_t)row[u + 1] > b) mine -= col[b - 1] > col[b];
    }
    const unsigned long long d = block_sum(mine, s_red);
    if (threadIdx.x == 0 && d) atomicAdd(descents, d);
}

// Hub-first order: each row's highest-degree neighbour (lowest id among
// ties) is swapped to the row's front, the neighbour a bottom-up step
// probes first.  One warp per row below HUB_CTA_ROW, one CTA above.
constexpr int HUB_CTA_ROW = 4096;

// deg: the rows' lengths (one 4-byte gather per entry instead of two offsets).
__device__ __forceinline__ unsigned long long hub_key(const int *__restrict__ deg, int v, int pos)
{
    return ((unsigned long long)(unsigned)__ldg(deg + v) << 32) | (unsigned)(0x7fffffff - pos);
}

template <typename RT>
__global__ void k_row_lengths(const RT *__restrict__ row, int n, int *deg)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        deg[v] = (int)(row[v + 1] - row[v]);
}

__device__ __forceinline__ void hub_swap(int *row_col, int pos)
{
    if (pos <= 0) return;
    const int t = row_col[0];
    row_col[0] = row_col[pos];
    row_col[pos] = t;
}

// A warp takes 32 consecutive rows: those of up to 8 entries a lane each, all
// at once, the others one after another (RMAT-22: 633 us with a warp per row and
// two offsets read per entry, 400 so).
template <typename RT>
__global__ void k_hub_first_warp(const RT *__restrict__ row, const int *__restrict__ deg, int n, int *col)
{
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = (int)lane_id();
    for (int64_t r0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; r0 < n; r0 += warps * 32) {
        const RT bl = r0 + lane < n ? row[r0 + lane] : 0;
        const int dl = r0 + lane < n ? deg[r0 + lane] : 0;
        if (dl >= 2 && dl <= 8) {
            int v[8];
            unsigned long long best = 0;
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = e < dl ? col[bl + e] : -1;
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (v[e] >= 0) {
                    const unsigned long long k = hub_key(deg, v[e], e);
                    best = k > best ? k : best;
                }
            hub_swap(col + bl, 0x7fffffff - (int)(best & 0xffffffffu));
        }
        unsigned left = __ballot_sync(FULL, dl > 8 && dl < HUB_CTA_ROW);
        while (left) {
            const int j = __ffs(left) - 1;
            left &= left - 1u;
            const RT b = __shfl_sync(FULL, bl, j);
            const int d = __shfl_sync(FULL, dl, j);
            unsigned long long best = 0;
#pragma unroll 4
            for (int i = lane; i < d; i += 32) {
                const unsigned long long k = hub_key(deg, col[b + i], i);
                best = k > best ? k : best;
            }
            // the longest length among the lanes, then its first place
            const unsigned top = __reduce_max_sync(FULL, (unsigned)(best >> 32));
            const unsigned at = __reduce_max_sync(FULL, (unsigned)(best >> 32) == top ? (unsigned)best : 0u);
            __syncwarp();
            if (lane == 0) hub_swap(col + b, 0x7fffffff - (int)at);
        }
    }
}

// Rows of HUB_GIANT_ROW entries or more: the whole grid splits each one.
constexpr int HUB_GIANT_ROW = 65536;

// Appends the rows of length in [lo, hi) to list (count in *cnt).
template <typename RT>
__global__ void k_rows_by_len(const RT *__restrict__ row, int n, int lo, int hi, int *list, unsigned *cnt)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        const int64_t r = base + lane_id();
        bool in = false;
        if (r < n) {
            const int64_t d = (int64_t)(row[r + 1] - row[r]);
            in = d >= lo && d < hi;
        }
        const unsigned m = __ballot_sync(FULL, in);
        if (!m) continue;
        unsigned pos = 0;
        if (lane_id() == 0) pos = atomicAdd(cnt, (unsigned)__popc(m));
        pos = __shfl_sync(FULL, pos, 0);
        if (in) list[pos + __popc(m & lanemask_lt())] = (int)r;
    }
}

// One CTA per listed row (list[0, *cnt)).
template <typename RT>
__global__ void k_hub_first_cta(const RT *__restrict__ row, const int *__restrict__ deg, const int *__restrict__ list, const unsigned *cnt, int *col)
{
    __shared__ unsigned long long s_best[32];
    const int count = (int)*cnt;
    for (int li = blockIdx.x; li < count; li += gridDim.x) {
        const int r = list[li];
        const RT b = row[r];
        const int d = (int)(row[r + 1] - b);
        unsigned long long best = 0;
        for (int i = threadIdx.x; i < d; i += blockDim.x) {
            const unsigned long long k = hub_key(deg, col[b + i], i);
            best = k > best ? k : best;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(FULL, best, o);
            best = y > best ? y : best;
        }
        if (lane_id() == 0) s_best[threadIdx.x >> 5] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (unsigned w = 1; w < (blockDim.x >> 5); w++) best = s_best[w] > best ? s_best[w] : best;
            const int pos = 0x7fffffff - (int)(best & 0xffffffffu);
            if (pos > 0) {
                const int t = col[b];
                col[b] = col[b + pos];
                col[b + pos] = t;
            }
        }
        __syncthreads();
    }
}

// The listed giant rows one after another, each split over the whole grid:
// every warp folds its entries' keys and takes the row's maximum with one
// atomicMax (best[g], zeroed by the caller); k_hub_giant_swap then moves it.
template <typename RT>
__global__ void k_hub_giant_max(const RT *__restrict__ row, const int *__restrict__ deg, const int *__restrict__ list, const unsigned *cnt,
                                const int *__restrict__ col, unsigned long long *best)
{
    const int count = (int)*cnt;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int g = 0; g < count; g++) {
        const int r = list[g];
        const RT b = row[r];
        const int d = (int)(row[r + 1] - b);
        unsigned long long mine = 0;
        for (int64_t i = tid; i < d; i += stride) {
            const unsigned long long k = hub_key(deg, col[b + i], (int)i);
            mine = k > mine ? k : mine;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(FULL, mine, o);
            mine = y > mine ? y : mine;
        }
        if (lane_id() == 0 && mine) atomicMax(best + g, mine);
    }
}

template <typename RT>
__global__ void k_hub_giant_swap(const RT *__restrict__ row, const int *__restrict__ list, const unsigned *cnt,
                                 const unsigned long long *best, int *col)
{
    const int count = (int)*cnt;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < count; g += gridDim.x * blockDim.x) {
        const RT b = row[list[g]];
        const int pos = 0x7fffffff - (int)(best[g] & 0xffffffffu);
        if (best[g] && pos > 0) {
            const int t = col[b];
            col[b] = col[b + pos];
            col[b + pos] = t;
        }
    }
}

int grid_for(int64_t work, int threads, int cap = 152 * 16)
{
    int64_t g = (work + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

struct Scratch {
    void *p = nullptr;
    ~Scratch() { if (p) cudaFree(p); }
};

// The block of c's vertex-sized arrays; row_bytes: room for row offsets in it,
// returned in row (0: none).
cudaError_t alloc_block(DeviceCsr &c, bool second, size_t row_bytes, void **row)
{
    const size_t n4 = sizeof(int) * (size_t)std::max(1, c.n);
    Carve cv;
    const size_t zmask = cv.add(sizeof(unsigned) * (((size_t)c.n + 31) / 32)), heavy = cv.add(n4), first = cv.add(n4);
    const size_t sec = second ? cv.add(n4) : 0, rows = row_bytes ? cv.add(row_bytes) : 0;
    const cudaError_t e = cudaMalloc(&c.block, cv.size);
    if (e != cudaSuccess) {
        c.block = nullptr;
        return e;
    }
    char *p = (char *)c.block;
    c.zmask = (unsigned *)(p + zmask);
    c.heavy = (int *)(p + heavy);
    c.first = (int *)(p + first);
    c.second = second ? (int *)(p + sec) : nullptr;
    if (row_bytes) *row = p + rows;
    return cudaSuccess;
}

template <typename RT>
int finalize_t(DeviceCsr &out, const RT *row, cudaStream_t st, std::string &err)
{
    int rc = GBFS_OK;
    struct Res {
        unsigned long long nonisolated;
        int maxdeg;
        unsigned nheavy, nover4, pad;
        unsigned long long part[SMALL_CTAS];
    };
    Pinned<Res> h;
    NEED_PINNED(h);
    Res *d_res = nullptr;
    const int W = (out.n + 31) / 32;
    CK(cudaMalloc(&d_res, sizeof(Res)));
    CK(cudaMemsetAsync(d_res, 0, sizeof(Res), st));
    static_assert(SMALL_MAX_N <= 256 * 152 * 16, "one pass of k_finalize's grid covers a small graph");
    if (out.n <= SMALL_MAX_N)
        k_finalize<true><<<grid_for((int64_t)W * 32, 256), 256, 0, st>>>(
            row, out.n, out.zmask, &d_res->maxdeg, &d_res->nonisolated, &d_res->nover4, d_res->part, small_part_log(out.n));
    else
        k_finalize<false><<<grid_for((int64_t)W * 32, 256), 256, 0, st>>>(
            row, out.n, out.zmask, &d_res->maxdeg, &d_res->nonisolated, &d_res->nover4, d_res->part, 0);
    CK(cudaGetLastError());
    k_heavy_list<<<grid_for(out.n, 1024, 152 * 4), 1024, 0, st>>>(row, out.n, out.heavy, &d_res->nheavy);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(h.p, d_res, sizeof(Res), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    out.max_degree = h->maxdeg;
    out.nonisolated = (int64_t)h->nonisolated;
    out.nover4 = (int32_t)h->nover4;
    out.nheavy = (int32_t)h->nheavy;
    out.part_cost = (int64_t)*std::max_element(h->part, h->part + SMALL_CTAS);
done:
    if (rc) cudaStreamSynchronize(st);  // before h's slot is another's
    if (d_res) cudaFree(d_res);
    return rc;
}

int finalize(DeviceCsr &out, cudaStream_t st, std::string &err)
{
    return out.wide ? finalize_t(out, (const long long *)out.row64, st, err)
                    : finalize_t(out, (const int *)out.row, st, err);
}

// The per-row sorts of one column array: lists by length, then one launch per
// length class.  The lists and the long rows' scratch are freed with it.
template <typename RT>
struct RowSorter {
    void *long_mem = nullptr;  // long rows: chunks and their counts
    int *tmp2 = nullptr;       // long rows: the merges' second place
    BinLists lists{};
    BinCounts *d_cnt = nullptr;
    Pinned<BinCounts> h;       // d_cnt's values once st has been synchronised
    Chunk *chunks = nullptr;
    int *ccnt = nullptr;
    bool bitmaps = false;      // the long rows have been sorted by k_long_rows

    ~RowSorter()
    {
        drop_tmp2();
        if (long_mem) cudaFree(long_mem);
    }

    // The sorts are done: room for the compacted columns.
    void drop_tmp2()
    {
        if (tmp2) cudaFree(tmp2);
        tmp2 = nullptr;
    }

    // Bytes of scratch the lists take (bin's mem) for n rows of m entries together.
    static size_t list_bytes(int32_t n, int64_t m)
    {
        int64_t cap[BIN_CLASSES];
        return 256 + sizeof(int) * (size_t)list_caps(n, m, cap);
    }
    static int64_t list_caps(int32_t n, int64_t m, int64_t (&cap)[BIN_CLASSES])
    {
        static const int over[BIN_CLASSES] = {32, W4_MAX, W16_MAX, 1024, 2048, MED_MAX};
        int64_t total = 0;
        for (int c = 0; c < BIN_CLASSES; c++) {
            cap[c] = std::min<int64_t>(n, m / (over[c] + 1)) + 1;
            total += cap[c];
        }
        return total;
    }

    // Lists by length; enqueued on st.  mem stays in use until the sorts are done.
    cudaError_t bin(const RT *row, int32_t n, int64_t m, void *mem, cudaStream_t st)
    {
        int64_t cap[BIN_CLASSES];
        list_caps(n, m, cap);
        d_cnt = (BinCounts *)mem;
        int *p = (int *)((char *)mem + 256);
        for (int c = 0; c < BIN_CLASSES; c++) {
            lists.list[c] = p;
            p += cap[c];
        }
        cudaError_t e = cudaSuccess;
        e = cudaMemsetAsync(mem, 0, 256, st);
        if (e != cudaSuccess) return e;
        k_bin<RT><<<grid_for(n, BIN_THREADS, 152 * 4), BIN_THREADS, 0, st>>>(row, n, lists, d_cnt);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h.p, d_cnt, sizeof(BinCounts), cudaMemcpyDeviceToHost, st);
        return e;
    }

    // The rows of list c by k_long_rows, where they may; taken: they are sorted.
    cudaError_t sort_long(int c, const RT *row, int32_t n, int *tmp, int *ucnt, cudaStream_t st, bool &taken)
    {
        taken = false;
        const BitmapShape shape(n);
        if (shape.ctas > BMR_CTAS) return cudaSuccess;
        static LaunchSetup setup;  // per row offset type
        auto config = [&](int ctas, int clusters, size_t smem, cudaLaunchAttribute *at) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(ctas * clusters));
            cfg.blockDim = dim3(BMR_THREADS);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st;
            at->id = cudaLaunchAttributeClusterDimension;
            at->val.clusterDim.x = (unsigned)ctas;
            at->val.clusterDim.y = at->val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            return cfg;
        };
        int sms = 0, fits = 0;
        cudaError_t e = setup.get(sms, fits, [&](int dev, int &s_out, int &f_out) {
            const size_t most = sizeof(unsigned) * BMR_THREADS * BMR_WORDS;
            cudaError_t x = cudaFuncSetAttribute(k_long_rows<RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
            if (x == cudaSuccess) x = cudaDeviceGetAttribute(&s_out, cudaDevAttrMultiProcessorCount, dev);
            cudaLaunchAttribute at;
            const cudaLaunchConfig_t cfg = config(BMR_CTAS, 1, most, &at);
            if (x == cudaSuccess) x = cudaOccupancyMaxActiveClusters(&f_out, k_long_rows<RT>, &cfg);
            return x;
        });
        if (e != cudaSuccess || fits < 1) {
            (void)cudaGetLastError();
            return cudaSuccess;
        }
        const int clusters = std::min((int)h->rows[c], std::max(1, BMR_CLUSTERS * sms / shape.ctas));
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = config(shape.ctas, clusters, shape.smem(), &at);
        e = cudaLaunchKernelEx(&cfg, k_long_rows<RT>, row, (const int *)lists.list[c],
                               (const unsigned *)(d_cnt->rows + c), shape.words, tmp, ucnt);
        taken = e == cudaSuccess;
        return e;
    }

    // Sorts the rows of tmp (the caller has synchronised st since bin).  Rows
    // are packed in place and counted in ucnt (n entries), distinct values only
    // with dedup; then the long rows' are left for compact().
    // spare (may be null): spare_n entries of scratch.
    cudaError_t sort(const RT *row, int32_t n, int *tmp, int dedup, int *ucnt, int *spare, int64_t spare_n,
                     cudaStream_t st)
    {
        const unsigned *rows = d_cnt->rows;
        const int thr = 256;
        cudaError_t e = cudaSuccess;
        const int nch = (int)h->chunks;
        if (nch && dedup) {
            e = sort_long(BIN_LONG, row, n, tmp, ucnt, st, bitmaps);
            if (e != cudaSuccess) return e;
            if (bitmaps) tl_route |= BUILD_LONG_BITS;
        }
        if (nch && !bitmaps) {
            const size_t cb = sizeof(Chunk) * (size_t)nch;
            e = cudaMalloc(&long_mem, 256 + cb + sizeof(int) * (size_t)nch);
            if ((int64_t)h->long_entries > spare_n) spare = nullptr;
            if (e == cudaSuccess && !spare) e = cudaMalloc(&tmp2, sizeof(int) * (size_t)h->long_entries);
            int *const two = spare ? spare : tmp2;
            if (e != cudaSuccess) return e;
            ChunkNext *next = (ChunkNext *)long_mem;
            chunks = (Chunk *)((char *)long_mem + 256);
            ccnt = (int *)((char *)long_mem + 256 + cb);
            e = cudaMemsetAsync(next, 0, sizeof(ChunkNext), st);
            if (e == cudaSuccess) e = cudaMemsetAsync(ucnt, 0, sizeof(int) * (size_t)n, st);
            if (e != cudaSuccess) return e;
            const int nl = (int)h->rows[BIN_LONG];
            const int grid = std::min(nch, 152 * 32);
            k_chunks<RT><<<grid_for(nl, 128), 128, 0, st>>>(row, lists.list[BIN_LONG], rows + BIN_LONG, chunks, next);
            k_sort_chunks<RT><<<grid, MED_THREADS, 0, st>>>(row, chunks, nch, tmp, two);
            const int passes = merge_passes(h->longest);
            for (int p = 0; p < passes; p++) k_merge<RT><<<grid, MED_THREADS, 0, st>>>(row, chunks, nch, tmp, two, p);
            if (dedup) k_chunk_unique<RT><<<grid, MED_THREADS, 0, st>>>(row, chunks, nch, tmp, ccnt, ucnt);
        }
        auto ctas = [](unsigned rows_, int cap) { return std::max(1, std::min((int)rows_, cap)); };
        bool done4k = false;
        if (h->rows[BIN_4K] && dedup && BitmapShape(n).ctas <= BMR_CTAS_4K)
            e = sort_long(BIN_4K, row, n, tmp, ucnt, st, done4k);
        if (e != cudaSuccess) return e;
        if (done4k) tl_route |= BUILD_4K_BITS;
        if (h->rows[BIN_4K] && !done4k)
            k_sort_block<512, RT><<<ctas(h->rows[BIN_4K], 152 * 16), 512, 0, st>>>(row, lists.list[BIN_4K],
                                                                                 rows + BIN_4K, tmp, dedup, ucnt);
        if (h->rows[BIN_2K])
            k_sort_block<256, RT><<<ctas(h->rows[BIN_2K], 152 * 32), 256, 0, st>>>(row, lists.list[BIN_2K],
                                                                                 rows + BIN_2K, tmp, dedup, ucnt);
        if (h->rows[BIN_1K])
            k_sort_block<128, RT><<<ctas(h->rows[BIN_1K], 152 * 64), 128, 0, st>>>(row, lists.list[BIN_1K],
                                                                                 rows + BIN_1K, tmp, dedup, ucnt);
        if (h->rows[BIN_W16])
            k_sort_warp<16, RT><<<152 * 8, 256, 0, st>>>(row, lists.list[BIN_W16], rows + BIN_W16, tmp, dedup, ucnt);
        if (h->rows[BIN_W4])
            k_sort_warp<4, RT><<<152 * 8, 256, 0, st>>>(row, lists.list[BIN_W4], rows + BIN_W4, tmp, dedup, ucnt);
        k_sort_small<RT><<<grid_for((int64_t)n * 32, thr), thr, 0, st>>>(row, n, tmp, dedup, ucnt);
        return cudaGetLastError();
    }

    // The long rows' distinct values into col (row2: the offsets there).
    cudaError_t compact(const RT *row, const RT *row2, const int *tmp, int *col, cudaStream_t st)
    {
        if (!h->chunks) return cudaSuccess;
        if (bitmaps) {
            const int tiles = (h->longest + CPL_THREADS * CPL_PER - 1) / (CPL_THREADS * CPL_PER);
            const dim3 grid(h->rows[BIN_LONG], (unsigned)std::min(tiles, 8));
            k_compact_long<RT><<<grid, CPL_THREADS, 0, st>>>(row, row2, lists.list[BIN_LONG], tmp, col);
            return cudaGetLastError();
        }
        k_compact_chunks<RT><<<std::min((int)h->chunks, 152 * 32), MED_THREADS, 0, st>>>(row, row2, chunks, (int)h->chunks,
                                                                                       ccnt, tmp, col);
        return cudaGetLastError();
    }
};

// Sort every row of (row, col) in place (no dedup).  Scratch is allocated
// and freed here.  Synchronises st.
template <typename RT>
int sort_rows_inplace(const RT *row, int *col, int32_t n, int64_t m, cudaStream_t st, std::string &err)
{
    int rc = GBFS_OK;
    char *mem = nullptr;
    RowSorter<RT> sorter;
    NEED_PINNED(sorter.h);
    Carve cv;
    const size_t ucnt = cv.add(sizeof(int) * ((size_t)n + 1)), lists = cv.add(sorter.list_bytes(n, m));
    CK(cudaMalloc(&mem, cv.size));
    CK(sorter.bin(row, n, m, mem + lists, st));
    CK(cudaStreamSynchronize(st));
    CK(sorter.sort(row, n, col, 0, (int *)(mem + ucnt), nullptr, 0, st));
    CK(cudaStreamSynchronize(st));
done:
    if (rc) cudaStreamSynchronize(st);  // before the sorter's slot is another's
    if (mem) cudaFree(mem);
    return rc;
}

// Hub-first order for every row of (row, col), m entries: one warp per row
// below HUB_CTA_ROW entries, one CTA per listed row up to HUB_GIANT_ROW,
// the whole grid per longer row (the few longest rows of a power-law
// graph would otherwise each hold one CTA for most of the pass).
// Synchronises st.
template <typename RT>
int hub_first_rows(const RT *row, int n, int64_t m, int *col, cudaStream_t st, std::string &err)
{
    int rc = GBFS_OK;
    char *mem = nullptr;
    int *deg = nullptr, *lists = nullptr;
    unsigned *cnts = nullptr;
    unsigned long long *best = nullptr;
    struct Counts {
        unsigned rows[2];  // long, giant
    };
    Pinned<Counts> h;
    NEED_PINNED(h);
    const int64_t cap_long = std::min<int64_t>(n, m / HUB_CTA_ROW + 1);
    const int64_t cap_giant = std::min<int64_t>(n, m / HUB_GIANT_ROW + 1);
    Carve cv;
    const size_t at_deg = cv.add(sizeof(int) * (size_t)n), at_lists = cv.add(sizeof(int) * (size_t)(cap_long + cap_giant)),
                 at_cnts = cv.add(2 * sizeof(unsigned));
    CK(cudaMalloc(&mem, cv.size));
    deg = (int *)(mem + at_deg);
    lists = (int *)(mem + at_lists);
    cnts = (unsigned *)(mem + at_cnts);
    CK(cudaMemsetAsync(cnts, 0, 2 * sizeof(unsigned), st));
    k_row_lengths<RT><<<grid_for(n, 256), 256, 0, st>>>(row, n, deg);
    k_hub_first_warp<RT><<<grid_for(n, 256, 152 * 64), 256, 0, st>>>(row, deg, n, col);
    CK(cudaGetLastError());
    k_rows_by_len<RT><<<grid_for(n, 256), 256, 0, st>>>(row, n, HUB_CTA_ROW, HUB_GIANT_ROW, lists, cnts);
    CK(cudaGetLastError());
    k_rows_by_len<RT><<<grid_for(n, 256), 256, 0, st>>>(row, n, HUB_GIANT_ROW, INT_MAX, lists + cap_long, cnts + 1);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(h.p, cnts, sizeof(Counts), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (h->rows[0]) {
        k_hub_first_cta<RT><<<152 * 2, 512, 0, st>>>(row, deg, lists, cnts, col);
        CK(cudaGetLastError());
    }
    if (h->rows[1]) {
        CK(cudaMalloc(&best, sizeof(unsigned long long) * h->rows[1]));
        CK(cudaMemsetAsync(best, 0, sizeof(unsigned long long) * h->rows[1], st));
        k_hub_giant_max<RT><<<152 * 4, 512, 0, st>>>(row, deg, lists + cap_long, cnts + 1, col, best);
        CK(cudaGetLastError());
        k_hub_giant_swap<RT><<<1, 256, 0, st>>>(row, lists + cap_long, cnts + 1, best, col);
        CK(cudaGetLastError());
    }
    CK(cudaStreamSynchronize(st));
done:
    if (rc) cudaStreamSynchronize(st);  // before h's slot is another's
    if (mem) cudaFree(mem);
    if (best) cudaFree(best);
    return rc;
}

}  // namespace

int csr_check_symmetric(DeviceCsr &c, cudaStream_t st, bool &sym, std::string &err)
{
    int rc = GBFS_OK;
    unsigned long long *descents = nullptr, h_descents = 0;
    int *flags = nullptr, *copy = nullptr;
    int h[2] = {0, 0};
    const int grid = grid_for(std::max<int64_t>(c.n, c.m), 256, 152 * 8);
    CK(cudaMalloc(&descents, 16));
    flags = (int *)(descents + 1);
    CK(cudaMemsetAsync(descents, 0, 16, st));
    if (!c.sorted_rows) {
        if (c.wide) k_check_sorted<<<grid, 256, 0, st>>>((const long long *)c.row64, c.col, c.n, c.m, descents);
        else k_check_sorted<<<grid, 256, 0, st>>>((const int *)c.row, c.col, c.n, c.m, descents);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&h_descents, descents, 8, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        c.sorted_rows = h_descents == 0;
    }
    {
        const int *col = c.col;
        if (!c.sorted_rows) {  // hub-first rows, for instance: check a sorted copy
            CK(cudaMalloc(&copy, sizeof(int) * (size_t)std::max<int64_t>(c.m, 1)));
            CK(cudaMemcpyAsync(copy, c.col, sizeof(int) * (size_t)c.m, cudaMemcpyDeviceToDevice, st));
            rc = c.wide ? sort_rows_inplace((const long long *)c.row64, copy, c.n, c.m, st, err)
                        : sort_rows_inplace((const int *)c.row, copy, c.n, c.m, st, err);
            if (rc) goto done;
            col = copy;
        }
        const int rows = grid_for(c.n, 256, 152 * 8);
        const bool by_rows = c.nheavy == 0;
        if (c.wide && by_rows) k_check_sym_rows<<<rows, 256, 0, st>>>((const long long *)c.row64, col, c.n, flags);
        else if (c.wide) k_check_sym<<<grid, 256, 0, st>>>((const long long *)c.row64, col, c.n, c.m, flags);
        else if (by_rows) k_check_sym_rows<<<rows, 256, 0, st>>>((const int *)c.row, col, c.n, flags);
        else k_check_sym<<<grid, 256, 0, st>>>((const int *)c.row, col, c.n, c.m, flags);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(h, flags, 8, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        sym = h[1] == 0;
    }
done:
    if (descents) cudaFree(descents);
    if (copy) cudaFree(copy);
    return rc;
}

int csr_hub_first(DeviceCsr &c, cudaStream_t st, std::string &err)
{
    int rc = GBFS_OK;
    rc = c.wide ? hub_first_rows((const long long *)c.row64, c.n, c.m, c.col, st, err)
                : hub_first_rows((const int *)c.row, c.n, c.m, c.col, st, err);
    if (rc) goto done;
    c.hub_rows = true;
    c.sorted_rows = false;
done:
    return rc;
}

namespace {

__global__ void k_in_count(const int *__restrict__ col, int64_t m, int *indeg)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&indeg[col[i]], 1);
}

// first[v] / second[v]: row v's first / second entry, -1 past its end
// (second may be null).
template <typename RT>
__global__ void k_first(const RT *__restrict__ row, const int *__restrict__ col, int n, int *first, int *second)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const RT b = row[v];
        const int d = (int)(row[v + 1] - b);
        first[v] = d > 0 ? col[b] : -1;
        if (second) second[v] = d > 1 ? col[b + 1] : -1;
    }
}

// Every out-edge u -> v lands in v's in-row (a warp per row took 610 us where
// one hub of 40 K edges sat among 4.8 M).
__global__ void k_in_scatter(const int *__restrict__ row, const int *__restrict__ col, int n, int64_t m, int *cursor,
                             int *tcol)
{
    for_edges(row, n, m, [&](int64_t e, int u, bool in) {
        if (in) tcol[atomicAdd(&cursor[col[e]], 1)] = u;
        return false;
    });
}

}  // namespace

int csr_build_transpose(DeviceCsr &c, cudaStream_t st, std::string &err)
{
    if (c.trow) return GBFS_OK;
    if (c.wide) {
        err = "no transpose of a graph with 64-bit row offsets (its searches stay top-down)";
        return GBFS_ERR_TOO_LARGE;
    }
    int rc = GBFS_OK;
    const int n = c.n;
    const int64_t m = c.m;
    int *indeg = nullptr, *cursor = nullptr, *trow = nullptr, *tcol = nullptr, *theavy = nullptr, *tfirst = nullptr;
    unsigned *d_nheavy = nullptr, h_nheavy = 0;
    void *scan_mem = nullptr;
    ScanScratch ss;
    const int64_t tiles = scan_tiles((int64_t)n + 1);
    CK(cudaMalloc(&indeg, sizeof(int) * ((size_t)n + 1)));
    CK(cudaMalloc(&trow, sizeof(int) * ((size_t)n + 1)));
    CK(cudaMalloc(&cursor, sizeof(int) * ((size_t)n + 1)));
    CK(cudaMalloc(&tcol, sizeof(int) * (size_t)std::max<int64_t>(m, 1)));
    CK(cudaMalloc(&theavy, sizeof(int) * (size_t)std::max(1, n)));
    CK(cudaMalloc(&tfirst, sizeof(int) * (size_t)std::max(1, n)));
    CK(cudaMalloc(&d_nheavy, sizeof(unsigned)));
    CK(cudaMemsetAsync(d_nheavy, 0, sizeof(unsigned), st));
    CK(cudaMalloc(&scan_mem, scan_scratch_bytes(tiles)));
    CK(cudaMemsetAsync(scan_mem, 0, scan_scratch_bytes(tiles), st));
    scan_scratch_carve(scan_mem, tiles, ss);
    CK(cudaMemsetAsync(indeg, 0, sizeof(int) * ((size_t)n + 1), st));
    if (m > 0) {
        k_in_count<<<grid_for(m, 256), 256, 0, st>>>(c.col, m, indeg);
        CK(cudaGetLastError());
    }
    CK(scan_exclusive_i32_i32(indeg, trow, n, trow + n, ss, st));
    CK(cudaMemcpyAsync(cursor, trow, sizeof(int) * ((size_t)n + 1), cudaMemcpyDeviceToDevice, st));
    if (m > 0) {
        k_in_scatter<<<grid_for(m, 256), 256, 0, st>>>(c.row, c.col, n, m, cursor, tcol);
        CK(cudaGetLastError());
    }
    k_heavy_list<<<grid_for(n, 1024, 152 * 4), 1024, 0, st>>>((const int *)trow, n, theavy, d_nheavy);
    CK(cudaGetLastError());
    // in-rows hub-first (the in-neighbour of highest in-degree, the likeliest
    // to be reached early, is probed first), then their first entries
    rc = hub_first_rows((const int *)trow, n, m, tcol, st, err);
    if (rc) goto done;
    k_first<<<grid_for(n, 256), 256, 0, st>>>((const int *)trow, (const int *)tcol, n, tfirst, (int *)nullptr);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&h_nheavy, d_nheavy, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    {
        unsigned h_scan_status[3] = {0, 0, 0};
        CK(cudaMemcpyAsync(h_scan_status, ss.ctl, 12, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (h_scan_status[2] != 0) {
            err = "scan look-back timed out";
            rc = GBFS_ERR_TIMEOUT;
            goto done;
        }
    }
    c.trow = trow;
    c.tcol = tcol;
    c.theavy = theavy;
    c.ntheavy = (int32_t)h_nheavy;
    c.tfirst = tfirst;
    trow = tcol = theavy = tfirst = nullptr;
done:
    if (theavy) cudaFree(theavy);
    if (tfirst) cudaFree(tfirst);
    if (d_nheavy) cudaFree(d_nheavy);
    if (indeg) cudaFree(indeg);
    if (cursor) cudaFree(cursor);
    if (trow) cudaFree(trow);
    if (tcol) cudaFree(tcol);
    if (scan_mem) cudaFree(scan_mem);
    return rc;
}

int csr_build_first(DeviceCsr &c, cudaStream_t st, std::string &err)
{
    int rc = GBFS_OK;
    // (hub-first rows are probed at their first entry alone: no second array)
    if (c.n > 0) {
        if (c.wide)
            k_first<<<grid_for(c.n, 256), 256, 0, st>>>((const long long *)c.row64, (const int *)c.col, c.n, c.first,
                                                        c.second);
        else
            k_first<<<grid_for(c.n, 256), 256, 0, st>>>((const int *)c.row, (const int *)c.col, c.n, c.first,
                                                        c.second);
        CK(cudaGetLastError());
    }
    CK(cudaStreamSynchronize(st));
done:
    return rc;
}

namespace {

template <typename RT>
__global__ void k_quads(const RT *__restrict__ row, const int *__restrict__ col, int n, int4 *quad, int *over,
                        unsigned *nover)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const RT b = row[v];
        const int d = (int)(row[v + 1] - b);
        int4 q = make_int4(-1, -1, -1, -1);
        if (d > 0) q.x = col[b];
        if (d > 1) q.y = col[b + 1];
        if (d > 2) q.z = col[b + 2];
        if (d == 4) q.w = col[b + 3];
        if (d > 4) {
            const unsigned k = atomicAdd(nover, 1u);
            q.w = -2 - (int)k;
            int *o = over + 16 * (size_t)k;
            for (int i = 0; i < 15; i++) o[i] = 3 + i < d ? col[b + 3 + i] : -1;
            o[15] = d;
        }
        quad[v] = q;
    }
}

}  // namespace

namespace {

// quad, over and the count of rows in over, in one allocation.
struct QuadLayout {
    Carve cv;
    size_t quad, over, cnt;
    explicit QuadLayout(const DeviceCsr &c)
    {
        quad = cv.add(sizeof(int4) * (size_t)std::max(1, c.n));
        over = cv.add(16 * sizeof(int) * (size_t)c.nover4);
        cnt = cv.add(sizeof(unsigned));
    }
};

}  // namespace

int64_t csr_quad_bytes(const DeviceCsr &c) { return (int64_t)QuadLayout(c).cv.size; }

int csr_build_quads(DeviceCsr &c, cudaStream_t st, std::string &err)
{
    if (c.quad) return GBFS_OK;
    int rc = GBFS_OK;
    char *mem = nullptr;
    const QuadLayout at(c);
    CK(cudaMalloc(&mem, at.cv.size));
    CK(cudaMemsetAsync(mem + at.cnt, 0, sizeof(unsigned), st));
    {
        int4 *const quad = (int4 *)(mem + at.quad);
        int *const over = (int *)(mem + at.over);
        unsigned *const cnt = (unsigned *)(mem + at.cnt);
        if (c.wide) k_quads<<<grid_for(c.n, 256), 256, 0, st>>>((const long long *)c.row64, c.col, c.n, quad, over, cnt);
        else k_quads<<<grid_for(c.n, 256), 256, 0, st>>>((const int *)c.row, c.col, c.n, quad, over, cnt);
        CK(cudaGetLastError());
        c.quad = quad;
        c.over = over;
    }
    mem = nullptr;
done:
    if (mem) cudaFree(mem);
    return rc;
}

void csr_drop_quads(DeviceCsr &c)
{
    if (c.quad) cudaFree(c.quad);
    c.quad = nullptr;
    c.over = nullptr;
}

int64_t csr_device_bytes(const DeviceCsr &c)
{
    const int64_t n = c.n, m = c.m;
    int64_t b = (c.wide ? 8 : 4) * (n + 1) + 4 * m + 4 * ((n + 31) / 32) + 4 * n;  // row, col, zmask, heavy list
    if (c.first) b += 4 * n;
    if (c.second) b += 4 * n;
    b += c.pieces_bytes;
    if (c.trow) b += 4 * (n + 1 + m) + 4 * n;                    // trow, tcol, theavy
    if (c.tfirst) b += 4 * n;
    if (c.quad) b += csr_quad_bytes(c);
    return b;
}

void csr_free(DeviceCsr &c)
{
    if (c.trow) cudaFree(c.trow);
    if (c.tcol) cudaFree(c.tcol);
    if (c.theavy) cudaFree(c.theavy);
    if (c.tfirst) cudaFree(c.tfirst);
    if (c.tpieces) cudaFree(c.tpieces);
    csr_drop_quads(c);
    if (c.pieces) cudaFree(c.pieces);
    if (c.own_row && c.row) cudaFree(c.row);
    if (c.own_row && c.row64) cudaFree(c.row64);
    if (c.col) cudaFree(c.col);
    if (c.block) cudaFree(c.block);
    if (c.keep) cudaFree(c.keep);
    c = DeviceCsr{};
}

namespace {

inline cudaError_t scan_rows(const int *in, int *out, int64_t n, ScanScratch &ss, cudaStream_t st)
{
    return scan_exclusive_i32_i32(in, out, n, out + n, ss, st);
}
inline cudaError_t scan_rows(const int *in, long long *out, int64_t n, ScanScratch &ss, cudaStream_t st)
{
    return scan_exclusive_i32_i64(in, out, n, out + n, ss, st);
}

// Memory for a build by buckets: the entries (words, then the columns before
// deduplication) and spare ones, for the overfull buckets and, as far as it
// goes, the long rows' second place.  Without packed: no buckets.
struct Buckets {
    BucketPlan *plan = nullptr;  // the caller's
    unsigned *packed = nullptr;
    int *spare = nullptr;
    int64_t spare_n = 0;

    bool take(int64_t md, int64_t over)
    {
        spare_n = std::max<int64_t>(over, md / 5 + 1);
        if (cudaMalloc(&packed, sizeof(unsigned) * (size_t)md) == cudaSuccess &&
            cudaMalloc(&spare, sizeof(int) * (size_t)spare_n) == cudaSuccess)
            return true;
        cudaGetLastError();
        drop();
        return false;
    }
    void drop()
    {
        if (packed) cudaFree(packed);
        if (spare) cudaFree(spare);
        packed = nullptr;
        spare = nullptr;
        spare_n = 0;
    }
    ~Buckets() { drop(); }
};

// Scratch of build_rows: row fill counts, later the rows' distinct counts; the
// lists of the sorts; and, where deduplication leaves them behind, the rows and
// columns before it.
template <typename RT>
struct BuildScratch {
    size_t fill, lists, rows = 0, cols = 0, size;
    // (with_cols: the entries go straight to their rows, not by buckets)
    BuildScratch(int32_t n, int64_t md, bool dedup, bool with_cols = true)
    {
        const size_t row_bytes = sizeof(RT) * ((size_t)n + 1);
        Carve cv;
        fill = cv.add(row_bytes);
        lists = cv.add(RowSorter<RT>::list_bytes(n, md));
        if (dedup) {
            rows = cv.add(row_bytes);
            if (with_cols) cols = cv.add(sizeof(int) * (size_t)std::max<int64_t>(md, 1));
        }
        size = cv.size;
    }
};

// Steps 2-5 with row offsets of type RT (int, or long long for wide
// graphs): offsets from the degrees, scatter, per-row sort, dedup
// compaction.  md: edges before deduplication.  On success the offsets and
// columns are in row_out (n + 1, the caller's) and col_out.  scratch: of
// BuildScratch's size, or null to allocate it here.  With room for buckets
// (taken over), by those instead of by the degrees.
template <typename RT>
int build_rows(int32_t n, int64_t m, int64_t md, const int *d_src, const int *d_dst, unsigned flags,
               const int *deg, Buckets &bk, char *scratch, ScanScratch &ss, cudaStream_t st, RT *row_out, int *&col_out,
               int64_t &m_out, std::string &err)
{
    int rc = GBFS_OK;
    const bool dedup = flags & GBFS_DEDUP;
    const size_t row_bytes = sizeof(RT) * ((size_t)n + 1);
    char *mem = nullptr;
    int *tmp = nullptr, *col = nullptr;
    const int thr = 256;
    const bool buckets = bk.packed != nullptr;
    const BuildScratch<RT> sc(n, md, dedup, !buckets);
    RowSorter<RT> sorter;
    Pinned<RT> h_m2;
    NEED_PINNED(sorter.h);
    NEED_PINNED(h_m2);
    if (!scratch) {
        CK(cudaMalloc(&mem, sc.size));
        scratch = mem;
    }
    if (buckets) {
        tmp = (int *)bk.packed;  // laid out in place
        bk.packed = nullptr;
    } else if (!dedup) {
        CK(cudaMalloc(&tmp, sizeof(int) * (size_t)std::max<int64_t>(md, 1)));
    }
    {
        RT *const row = dedup ? (RT *)(scratch + sc.rows) : row_out;
        RT *const cursor = (RT *)(scratch + sc.fill);
        int *const ucnt = (int *)(scratch + sc.fill);
        int *const to = tmp ? tmp : (int *)(scratch + sc.cols);
        if (buckets) {
            int vbits = 1;
            while ((1 << vbits) < n) vbits++;
            CK(cudaFuncSetAttribute(k_bucket_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(BucketShared)));
            k_bucket_scatter<<<152, BK_SBLOCK, sizeof(BucketShared), st>>>(d_src, d_dst, m, n, flags, vbits, bk.plan,
                                                                          (int *)(scratch + sc.fill), (unsigned *)tmp);
            CK(cudaGetLastError());
            CK(cudaFuncSetAttribute(k_bucket_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(int) * BK_STAGE));
            if constexpr (sizeof(RT) == sizeof(int))
                k_bucket_rows<<<((n - 1) >> BK_LOG) + 1, BK_BLOCK, sizeof(int) * BK_STAGE, st>>>(
                    bk.plan, (unsigned *)tmp, vbits, n, row, bk.spare);
            CK(cudaGetLastError());
            CK(sorter.bin(row, n, md, scratch + sc.lists, st));
        } else {
            CK(scan_rows(deg, row, n, ss, st));
            CK(sorter.bin(row, n, md, scratch + sc.lists, st));
            CK(cudaMemcpyAsync(cursor, row, row_bytes, cudaMemcpyDeviceToDevice, st));
            if (m > 0) {
                k_scatter<RT><<<grid_for(m, thr, EDGE_CTAS), thr, 0, st>>>(d_src, d_dst, m, n, flags, cursor, to);
                CK(cudaGetLastError());
            }
        }
        CK(cudaStreamSynchronize(st));  // the sorter's counts are here

        // Per-row sort (+ distinct count).
        CK(sorter.sort(row, n, to, dedup, ucnt, bk.spare, bk.spare_n, st));

        if (dedup) {
            CK(scan_rows(ucnt, row_out, n, ss, st));
            CK(cudaMemcpyAsync(h_m2.p, row_out + n, sizeof(RT), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            sorter.drop_tmp2();
            bk.drop();
            CK(cudaMalloc(&col, sizeof(int) * (size_t)std::max<int64_t>((int64_t)*h_m2.p, 1)));
            k_compact<RT><<<grid_for((int64_t)n * 32, thr), thr, 0, st>>>(row, row_out, n, to, col);
            CK(cudaGetLastError());
            CK(sorter.compact(row, row_out, to, col, st));
            m_out = (int64_t)*h_m2.p;
        } else {
            col = tmp;
            tmp = nullptr;
            m_out = md;
        }
        CK(cudaStreamSynchronize(st));
    }
    col_out = col;
    col = nullptr;
done:
    if (rc) cudaStreamSynchronize(st);  // before the slots of h_m2 and the sorter are another's
    if (mem) cudaFree(mem);
    if (col) cudaFree(col);
    if (tmp) cudaFree(tmp);
    return rc;
}

}  // namespace

int csr_build_from_edges(int32_t n, int64_t m, const int *d_src, const int *d_dst, unsigned flags,
                         cudaStream_t st, DeviceCsr &out, std::string &err)
{
    int rc = GBFS_OK;
    char *mem = nullptr;
    int *deg = nullptr, *status = nullptr;
    unsigned long long *total = nullptr;
    ScanScratch ss;
    struct Counted {
        int status, pad;
        unsigned long long total;
        unsigned scan[3];
        unsigned long long bucket_total;
        unsigned bucket_largest, bucket_near, bucket_seen, bucket_over;
    };
    Buckets bk;
    Pinned<Counted> h;
    NEED_PINNED(h);
    const int thr = 256;
    out = DeviceCsr{};
    out.n = n;
    tl_route = 0;

    // Degrees, scratch for both scans (n+1 elements at most), and the counters.
    const int64_t tiles = scan_tiles((int64_t)n + 1);
    Carve cv;
    const size_t at_deg = cv.add(sizeof(int) * ((size_t)n + 1)), at_scan = cv.add(scan_scratch_bytes(tiles)),
                 at_status = cv.add(64), at_plan = cv.add(sizeof(BucketPlan));
    const size_t zeroed = cv.size;
    // with it the scratch of the steps after the count, sized by the input, if
    // that is small (a large one waits for the count, which may be smaller)
    const int64_t most = m * (flags & GBFS_SYMMETRIZE ? 2 : 1);
    const size_t later = flags & GBFS_WIDE_ROWS ? BuildScratch<long long>(n, most, flags & GBFS_DEDUP).size
                                                : BuildScratch<int>(n, most, flags & GBFS_DEDUP).size;
    const bool together = later <= (size_t)64 << 20;
    const size_t at_later = together ? cv.add(later) : 0;
    CK(cudaMalloc(&out.keep, 256));
    CK(cudaMalloc(&mem, cv.size));
    CK(cudaMemsetAsync(mem, 0, zeroed, st));
    scan_scratch_carve(mem + at_scan, tiles, ss);
    deg = (int *)(mem + at_deg);
    status = (int *)(mem + at_status);
    total = (unsigned long long *)(status + 2);
    bk.plan = (BucketPlan *)(mem + at_plan);
    if (!(flags & GBFS_WIDE_ROWS) && most >= BK_MIN_M && most <= INT32_MAX && n <= BK_MAX_N) {
        k_bucket_hist<<<152 * 2, BK_BLOCK, 0, st>>>(d_src, d_dst, m, n, flags, bk.plan, status);
        CK(cudaGetLastError());
        k_bucket_plan<<<1, BK_BLOCK, 0, st>>>(bk.plan, ((n - 1) >> BK_LOG) + 1);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&h->bucket_total, bk.plan, 24, cudaMemcpyDeviceToHost, st));  // total to over
        CK(cudaStreamSynchronize(st));
        // (no room for them: straight to the rows)
        if (h->bucket_largest <= BK_MAX_BUCKET && h->bucket_total > 0 && h->bucket_near <= h->bucket_seen / 2 &&
            bk.take((int64_t)h->bucket_total, h->bucket_over))
            CK(cudaMemcpyAsync(total, &bk.plan->total, 8, cudaMemcpyDeviceToDevice, st));
        if (bk.packed) tl_route |= BUILD_BUCKETS;
    }
    if (m > 0 && !bk.packed) {
        k_count<<<grid_for(m, thr, EDGE_CTAS), thr, 0, st>>>(d_src, d_dst, m, n, flags, deg, total, status);
        CK(cudaGetLastError());
    }
    CK(cudaMemcpyAsync(h.p, status, 16, cudaMemcpyDeviceToHost, st));  // status and total
    CK(cudaStreamSynchronize(st));
    if (h->status == DEV_OVERFLOW) {
        err = "a vertex with 2^30 or more edges";
        rc = GBFS_ERR_TOO_LARGE;
        goto done;
    }
    if (h->status != DEV_OK) {
        err = "edge endpoint outside [0, n)";
        rc = GBFS_ERR_INVALID_ARG;
        goto done;
    }
    out.wide = (flags & GBFS_WIDE_ROWS) || h->total > (unsigned long long)INT32_MAX;
    {
        const size_t row_bytes = (out.wide ? sizeof(long long) : sizeof(int)) * ((size_t)n + 1);
        void *row = nullptr;
        CK(alloc_block(out, !(flags & GBFS_HUB_FIRST), row_bytes, &row));
        if (out.wide) out.row64 = (long long *)row;
        else out.row = (int *)row;
    }
    {
        char *const later_mem = together ? mem + at_later : nullptr;
        const int64_t md = (int64_t)h->total;
        if (out.wide)
            rc = build_rows<long long>(n, m, md, d_src, d_dst, flags, deg, bk, later_mem, ss, st, out.row64, out.col,
                                       out.m, err);
        else
            rc = build_rows<int>(n, m, md, d_src, d_dst, flags, deg, bk, later_mem, ss, st, out.row, out.col, out.m, err);
    }
    if (rc) goto done;
    out.sorted_rows = true;
    CK(cudaMemcpyAsync(h->scan, ss.ctl, 12, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (h->scan[2] != 0) {
        err = "scan look-back timed out";
        rc = GBFS_ERR_TIMEOUT;
        goto done;
    }
    rc = finalize(out, st, err);

done:
    if (rc) cudaStreamSynchronize(st);  // before h's slot is another's
    if (mem) cudaFree(mem);
    if (rc != GBFS_OK) csr_free(out);
    return rc;
}

namespace {

template <typename RT>
int csr_adopt_t(int32_t n, int64_t m, RT *d_row, int *d_col, cudaStream_t st, DeviceCsr &out, std::string &err)
{
    int rc = GBFS_OK;
    int *status = nullptr;
    RT h[2] = {0, 0};
    int h_status = 0;
    CK(cudaMalloc(&out.keep, 256));
    CK(cudaMalloc(&status, sizeof(int)));
    CK(cudaMemsetAsync(status, 0, sizeof(int), st));
    k_validate_csr<RT><<<grid_for(std::max<int64_t>(m, n), 256), 256, 0, st>>>(d_row, d_col, n, m, status);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&h[0], d_row, sizeof(RT), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&h[1], d_row + n, sizeof(RT), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&h_status, status, 4, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (h[0] != 0 || (int64_t)h[1] != m || h_status != DEV_OK) {
        err = "CSR is not well formed (row_offset[0]==0, non-decreasing, row_offset[n]==m, "
              "col ids in [0, n))";
        rc = GBFS_ERR_INVALID_ARG;
        goto done;
    }
    CK(alloc_block(out, true, 0, nullptr));
    rc = finalize(out, st, err);
done:
    if (status) cudaFree(status);
    if (rc != GBFS_OK) csr_free(out);
    return rc;
}

}  // namespace

int csr_adopt(int32_t n, int64_t m, int *d_row, int *d_col, cudaStream_t st, DeviceCsr &out,
              std::string &err)
{
    out = DeviceCsr{};
    out.n = n;
    out.m = m;
    out.row = d_row;
    out.own_row = true;
    out.col = d_col;
    return csr_adopt_t(n, m, d_row, d_col, st, out, err);
}

int csr_adopt64(int32_t n, int64_t m, long long *d_row, int *d_col, cudaStream_t st, DeviceCsr &out,
                std::string &err)
{
    out = DeviceCsr{};
    out.n = n;
    out.m = m;
    out.row64 = d_row;
    out.own_row = true;
    out.wide = true;
    out.col = d_col;
    return csr_adopt_t(n, m, d_row, d_col, st, out, err);
}

}  // namespace gbfs
