// parents.cu -- BFS-tree parents from a finished level array (sm_103a).
//
// The reference's 2D CPU BFS keeps a predecessor per vertex, the frontier
// vertex that happened to discover it first (2D Partition/src/cpuBFS.cpp:16,56);
// its GPU counterpart (d_pred, 2D Partition/include/gpuBFS.cuh:45) inherits
// whatever order the threads ran in.  Here the parent is canonical:
//
//     parent[v] = min { u : edge u -> v, level[u] == level[v] - 1 }
//
// and -1 for the source and for unreached vertices, so one graph and source
// give one parent array and every entry is a valid BFS-tree parent.
//
// A vertex of level 1 has one possible parent, the source.  The others:
// symmetric graphs pull: each vertex looks for the smallest neighbour one
// level closer, in ascending rows up to the first hit (one thread per row of
// up to HEAVY_DEGREE entries, one warp per longer row, and the rows past
// MS_HUGE in pieces of MS_PIECE over all warps with an atomicMin per piece).
// Directed graphs push: every reached u offers itself to the out-neighbours
// one level further with atomicMin, after a plain-load filter (parent values
// only decrease), one warp per row or piece, up to 256 entries at once (a
// directed RMAT of 8 M entries: 295 us a call with 32, 215 so).  On large
// symmetric graphs with rows in other than ascending order, levels whose
// vertices have far more edges than the level before are pushed to as well.
//
// The longest rows bounded this: RMAT-20 with its search took 1,060 us with a
// warp to each row, walked to its end (900 of them in the heavy rows' kernel),
// and takes 145 to 155 us now; the level gathers hit L2.
#include <algorithm>
#include <climits>

#include "bfs.cuh"
#include "common.cuh"
#include "index.h"
#include "msbfs.cuh"
#include "parents.cuh"

namespace gbfs {

namespace {

constexpr int PT = 256;
constexpr int OFFER_ILP = 8;  // a lane's offers in flight in long rows
constexpr unsigned long long PUSH_SHARE = 4;
constexpr int64_t PUSH_MIN_M = 1 << 23;

__device__ __forceinline__ bool is_set(unsigned mask, int l) { return l < 32 && mask >> l & 1u; }

// Smallest entry u of row entries [b, e) with level[u] == want; INT_MAX if
// none.  The whole warp walks them, 128 a step; sorted: ascending entries,
// the first hit ends the walk.  All 32 lanes get the result.
template <typename RT>
__device__ __forceinline__ int warp_min_at(const int *__restrict__ col, RT b, RT e, const int *__restrict__ level,
                                           int want, bool sorted, int lane)
{
    int best = INT_MAX;
    for (RT i0 = b; idx_before(i0, e); i0 = idx_add(i0, 128)) {
        int u[4], l[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const RT i = idx_add(i0, t * 32 + lane);
            u[t] = idx_before(i, e) ? __ldg(col + i) : -1;
        }
#pragma unroll
        for (int t = 0; t < 4; t++) l[t] = u[t] >= 0 ? __ldg(level + u[t]) : -2;
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (l[t] == want) best = min(best, u[t]);
        if (sorted && __any_sync(FULL, best != INT_MAX)) break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(FULL, best, o));
    return best;
}

// Bit l: the vertices of level l + 1 get their parents offered by those of level
// l instead of looking for them, where level l has less than 1 / PUSH_SHARE of
// the edges of level l + 1.  From the search's trace; rows of several levels (of
// the label-correcting kernels) give no bit.  All threads call it.
__device__ __forceinline__ unsigned pushed_levels(const BfsCtrl *ctrl)
{
    __shared__ unsigned s_mask;
    if (threadIdx.x < 32) {
        const int l = (int)threadIdx.x, len = min(ctrl->trace_len, TRACE_CAP - 1);
        unsigned long long here = 0, next = 0;
        if (l >= 1 && l + 1 < len) {
            const LevelTrace a = ctrl->trace[l], b = ctrl->trace[l + 1];
            if (a.level == l && b.level == l + 1 && a.dir < 4 && b.dir < 4) {
                here = a.edges;
                next = b.edges;
            }
        }
        const unsigned m = __ballot_sync(FULL, here * PUSH_SHARE < next);
        if (l == 0) s_mask = m;
    }
    __syncthreads();
    return s_mask;
}

template <bool PUSH, typename RT>
__global__ void k_parents_pull_light(const RT *__restrict__ row, const int *__restrict__ col, int n, int source,
                                     bool sorted, const BfsCtrl *ctrl, const int *__restrict__ level,
                                     int *__restrict__ parent)
{
    const unsigned push = PUSH ? pushed_levels(ctrl) : 0u;
    for (long long v = (long long)blockIdx.x * PT + threadIdx.x; v < n; v += (long long)gridDim.x * PT) {
        const int lv = level[v];
        int best = lv == 1 ? source : -1;
        if (lv > 1) {
            best = INT_MAX;  // stays so for offers, and in a long row: the heavy kernel's
            const RT b = row[v], e = row[v + 1];
            if (e - b <= HEAVY_DEGREE && !is_set(push, lv - 1)) {
                for (RT i = b; idx_before(i, e); i = idx_add(i, 4)) {
                    int u[4], l[4];
#pragma unroll
                    for (int t = 0; t < 4; t++) u[t] = __ldg(col + idx_end(i, t, e - 1));
#pragma unroll
                    for (int t = 0; t < 4; t++) l[t] = __ldg(level + u[t]);
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (l[t] == lv - 1) best = min(best, u[t]);
                    if (sorted && best != INT_MAX) break;
                }
            }
        }
        parent[v] = best;
    }
}

// offer u, of level lu, to its out-neighbours [b, e) of the next level
template <int ILP, typename RT>
__device__ __forceinline__ void warp_offer_by(int u, int lu, const int *__restrict__ col, RT b, RT e,
                                              const int *__restrict__ level, int *parent, int lane)
{
    for (RT i0 = b; idx_before(i0, e); i0 = idx_add(i0, 32 * ILP)) {
        int v[ILP], l[ILP];
#pragma unroll
        for (int t = 0; t < ILP; t++) {
            const RT i = idx_add(i0, t * 32 + lane);
            v[t] = idx_before(i, e) ? __ldg(col + i) : -1;
        }
#pragma unroll
        for (int t = 0; t < ILP; t++) l[t] = v[t] >= 0 ? __ldg(level + v[t]) : -2;
#pragma unroll
        for (int t = 0; t < ILP; t++)
            if (l[t] == lu + 1) l[t] = ld_relaxed_i32(parent + v[t]);
            else l[t] = -1;
#pragma unroll
        for (int t = 0; t < ILP; t++)
            if (l[t] > u) atomicMin(parent + v[t], u);
    }
}

template <typename RT>
__device__ __forceinline__ void warp_offer(int u, int lu, const int *__restrict__ col, RT b, RT e,
                                           const int *__restrict__ level, int *parent, int lane)
{
    if (e - b <= 32) warp_offer_by<1>(u, lu, col, b, e, level, parent, lane);
    else if (e - b <= 64) warp_offer_by<2>(u, lu, col, b, e, level, parent, lane);
    else warp_offer_by<OFFER_ILP>(u, lu, col, b, e, level, parent, lane);
}

// Long rows, and the offers of all rows (see pushed_levels).
template <bool PUSH, typename RT>
__global__ void k_parents_pull_heavy(const RT *__restrict__ row, const int *__restrict__ col, int n,
                                     const int *__restrict__ heavy, int nheavy, const int2 *__restrict__ pieces,
                                     int npieces, bool sorted, const BfsCtrl *ctrl, const int *__restrict__ level,
                                     int *parent)
{
    const unsigned push = PUSH ? pushed_levels(ctrl) : 0u;
    const long long gw = ((long long)blockIdx.x * PT + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * PT) >> 5;
    const int lane = threadIdx.x & 31;
    for (long long c = gw; c < npieces; c += nw) {
        const int2 pc = __ldg(pieces + c);
        const int lv = __ldg(level + pc.x);
        if (lv < 1) continue;  // written by the light kernel, as is level 1
        const RT b = row[pc.x] + (RT)pc.y * MS_PIECE;
        const RT e = idx_end(b, MS_PIECE, row[pc.x + 1]);
        if (is_set(push, lv)) warp_offer(pc.x, lv, col, b, e, level, parent, lane);
        if (lv == 1 || is_set(push, lv - 1)) continue;
        // an earlier piece of an ascending row has the answer (one read,
        // broadcast: the branch is the warp's)
        if (sorted && __shfl_sync(FULL, ld_relaxed_i32(parent + pc.x), 0) <= __ldg(col + b)) continue;
        const int best = warp_min_at(col, b, e, level, lv - 1, sorted, lane);
        if (lane == 0 && best != INT_MAX) atomicMin(parent + pc.x, best);
    }
    for (long long h = gw; h < nheavy; h += nw) {
        const int v = __ldg(heavy + h);
        const int lv = __ldg(level + v);
        const RT b = row[v], e = row[v + 1];
        if (lv < 1 || (npieces > 0 && e - b > MS_HUGE)) continue;
        if (is_set(push, lv)) warp_offer(v, lv, col, b, e, level, parent, lane);
        if (lv == 1 || is_set(push, lv - 1)) continue;
        const int best = warp_min_at(col, b, e, level, lv - 1, sorted, lane);
        if (lane == 0) parent[v] = best;
    }
    if (!push) return;
    for (long long v0 = gw * 32; v0 < n; v0 += nw * 32) {
        const int mine = v0 + lane < n ? __ldg(level + v0 + lane) : -1;
        unsigned left = __ballot_sync(FULL, mine >= 1 && is_set(push, mine));
        while (left) {
            const int o = __ffs(left) - 1;
            left &= left - 1;
            const RT b = row[v0 + o], e = row[v0 + o + 1];
            if (e - b > HEAVY_DEGREE) continue;
            warp_offer((int)(v0 + o), __shfl_sync(FULL, mine, o), col, b, e, level, parent, lane);
        }
    }
}

__global__ void k_parents_init(int n, int source, const int *__restrict__ level, int *__restrict__ parent)
{
    for (long long v = (long long)blockIdx.x * PT + threadIdx.x; v < n; v += (long long)gridDim.x * PT)
        parent[v] = level[v] > 1 ? INT_MAX : level[v] == 1 ? source : -1;
}

template <typename RT>
__global__ void k_parents_push(const RT *__restrict__ row, const int *__restrict__ col, int n,
                               const int2 *__restrict__ pieces, int npieces, const int *__restrict__ level,
                               int *parent)
{
    const long long gw = ((long long)blockIdx.x * PT + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * PT) >> 5;
    const int lane = threadIdx.x & 31;
    for (long long c = gw; c < npieces; c += nw) {
        const int2 pc = __ldg(pieces + c);
        const int lu = __ldg(level + pc.x);
        if (lu < 1) continue;  // unreached, or the source (its offers are in place)
        const RT b = row[pc.x] + (RT)pc.y * MS_PIECE;
        warp_offer(pc.x, lu, col, b, idx_end(b, MS_PIECE, row[pc.x + 1]), level, parent, lane);
    }
    for (long long u = gw; u < n; u += nw) {
        const int lu = __ldg(level + u);
        if (lu < 1) continue;
        const RT b = row[u], e = row[u + 1];
        if (npieces > 0 && e - b > MS_HUGE) continue;
        warp_offer((int)u, lu, col, b, e, level, parent, lane);
    }
}

int grid_of(long long work, int cap)
{
    long long b = (work + PT - 1) / PT;
    return (int)std::max(1LL, std::min<long long>(b, cap));
}

}  // namespace

namespace {

template <typename RT>
cudaError_t parents_launch(const DeviceCsr &g, const RT *row, bool symmetric, int source, const int *d_level,
                           const BfsCtrl *ctrl, int *d_parent, cudaStream_t st)
{
    const int np = g.pieces ? g.npieces : 0;
    if (symmetric) {
        // Levels that are cheaper to push to are, where rows are not ascending
        // (RMAT-20, hub-first rows: whole call 227 us pulling all, 175 so;
        // RMAT-21 369 and 230; ascending rows end early when pulled: RMAT-20 143
        // and 174) and the graph is large (1.8 M entries: 98 and 102 us, 13 M:
        // 143 and 121).
        const int grid_l = grid_of(g.n, 152 * 16);
        if (!g.sorted_rows && g.nheavy > 0 && g.m >= PUSH_MIN_M) {
            k_parents_pull_light<true, RT><<<grid_l, PT, 0, st>>>(row, g.col, g.n, source, false, ctrl, d_level, d_parent);
            k_parents_pull_heavy<true, RT><<<152 * 16, PT, 0, st>>>(row, g.col, g.n, g.heavy, g.nheavy, g.pieces, np,
                                                                    false, ctrl, d_level, d_parent);
            return cudaGetLastError();
        }
        k_parents_pull_light<false, RT><<<grid_l, PT, 0, st>>>(row, g.col, g.n, source, g.sorted_rows, ctrl, d_level,
                                                               d_parent);
        if (g.nheavy > 0)
            k_parents_pull_heavy<false, RT><<<grid_of(((long long)g.nheavy + np) * 32, 152 * 16), PT, 0, st>>>(
                row, g.col, g.n, g.heavy, g.nheavy, g.pieces, np, g.sorted_rows, ctrl, d_level, d_parent);
    } else {
        k_parents_init<<<grid_of(g.n, 152 * 16), PT, 0, st>>>(g.n, source, d_level, d_parent);
        k_parents_push<RT><<<grid_of((long long)g.n * 32, 152 * 16), PT, 0, st>>>(row, g.col, g.n, g.pieces, np,
                                                                                 d_level, d_parent);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t parents_enqueue(const DeviceCsr &g, bool symmetric, int source, const int *d_level, const BfsCtrl *ctrl,
                            int *d_parent, cudaStream_t st)
{
    if (g.n == 0) return cudaSuccess;
    return g.wide ? parents_launch(g, (const long long *)g.row64, symmetric, source, d_level, ctrl, d_parent, st)
                  : parents_launch(g, (const int *)g.row, symmetric, source, d_level, ctrl, d_parent, st);
}

}  // namespace gbfs
