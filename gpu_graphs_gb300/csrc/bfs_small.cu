// bfs_small.cu -- single-source search of a small graph on one thread-block
// cluster (sm_103a).
//
// On a graph of some ten thousand vertices a search is a handful of levels of
// a few microseconds' work each, and the grid kernel (bfs.cu) spends its time
// on what separates them: a barrier over 304 CTAs, a queue through L2, and
// claims that are L2 atomics, one dependent round trip after another.  Here a
// cluster of up to 16 CTAs holds the whole search in its shared memory.  CTA c
// owns 2^LOGS consecutive vertices (row offsets, levels, visited bits) and has
// a bitmap over ALL vertices of its own to mark neighbours in.  Per level, a CTA
//   1. reads its vertices' words of every CTA's bitmap (distributed shared
//      memory, 16 bytes a load): its new vertices;
//   2. lists their rows;
//   3. walks those rows, a group of lanes per row (about half as wide as the
//      level's rows are long; the whole CTA on long ones), and marks each
//      neighbour in its own bitmap: the column entries are the level's only
//      global loads;
// and a cluster barrier ends the level.  Marking a neighbour at its owner
// instead, one remote reduction per edge, ran at an edge per six cycles and SM
// (65,536 vertices, 524 K edges: 125 us against 45).  Levels stay in shared memory to the end:
// a global store in the loop would make the barrier's release wait for it.
// Uniform random graphs, device time here and in the grid kernel: 1,000
// vertices 17 and 44 us, 65,536 vertices 45 and 91 us (top-down).  What is left
// is two or three thousand cycles a level: shared-memory steps in sequence, one
// column load, the barrier; and on levels of many edges the marks.
// Replaces, for such graphs, the per-level host loop of gpuBFS::gpuBFS
// (1D Partition/src/gpuBFS.cu:66-100).
#include <algorithm>

#include "bfs.cuh"
#include "bfs_args.cuh"
#include "blockq.cuh"

namespace gbfs {

namespace {

constexpr int SM_CTAS = SMALL_CTAS;  // CTAs of the largest cluster
constexpr int SM_LONG = SMALL_LONG;  // rows the whole CTA walks
constexpr int SM_TRACE = 64;     // trace rows held in shared memory

// The longest row is more than 16 times the mean one.
__host__ __device__ inline bool small_skewed(long long max_degree, long long n, long long m)
{
    return max_degree * n > 16 * m;
}

template <int LOGS>
struct SmallShared {
    static constexpr int S = 1 << LOGS;
    unsigned bits[2][SM_CTAS * S / 32];   // the neighbours this CTA marked, by level parity
    unsigned long long slot[2][SM_CTAS];  // each CTA's new vertices | their out-edges, by level parity
    unsigned long long trace[SM_TRACE][2];
    unsigned rows[2], longs[2], verts[2], degs[2];  // of the level: short and long rows, vertices, out-edges
    unsigned fresh[S / 32];               // this level's vertices
    unsigned visited[S / 32];
    int level[S];
    int row[S + 1];                       // row offsets (a small graph's fit 32 bits)
    int2 list[S];                         // the frontier's row bounds: short rows, and long ones from the end
};

template <int LOGS, int BLOCK, typename RT>
__global__ void __launch_bounds__(BLOCK, 1) k_bfs_small(BfsArgs a)
{
    constexpr int S = 1 << LOGS, PER = S / BLOCK, W = S / 32;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    auto &sh = *reinterpret_cast<SmallShared<LOGS> *>(sm_raw);
    const int t = (int)threadIdx.x;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const unsigned rank = cluster_rank(), ctas = cluster_size();
    const int n = a.n, base = (int)rank << LOGS;
    const int own = max(0, min(S, n - base));
    const RT *const row = RowSel<RT>::row(a);
    BfsCtrl *ctrl = a.ctrl;
    const bool head = rank == 0 && t == 0;
    if (head) ctrl->t_entry = globaltimer_ns();

    for (int i = t; i <= own; i += BLOCK) sh.row[i] = (int)__ldg(row + base + i);
    for (int i = t; i < (int)ctas * W; i += BLOCK) {
        sh.bits[0][i] = 0;
        sh.bits[1][i] = 0;
    }
    for (int i = t; i < W; i += BLOCK) {
        sh.fresh[i] = 0;
        sh.visited[i] = 0;
    }
    for (int i = t; i < S; i += BLOCK) sh.level[i] = -1;
    if (t < 2) sh.rows[t] = sh.longs[t] = sh.verts[t] = sh.degs[t] = 0;
    __syncthreads();
    if (a.single_root >= 0) {
        if (t == 0 && a.single_root >> LOGS == (int)rank) sh.bits[0][a.single_root >> 5] = 1u << (a.single_root & 31);
    } else {
        for (int i = t; i < a.nroots; i += BLOCK) {
            const int r = a.roots[i];
            if ((unsigned)r < (unsigned)n && r >> LOGS == (int)rank) atomicOr(&sh.bits[0][r >> 5], 1u << (r & 31));
        }
    }
    const bool alone = ctas == 1;
    // groups twice as wide where row lengths differ much (RMAT, 65,536 vertices,
    // 740 K edges: 55 us without, 52 with; uniform random, 524 K: 45 and 48)
    const int skewed = small_skewed(a.max_degree, a.n, a.m) ? 1 : 0;
    if (alone) __syncthreads();
    else cluster_barrier();
    if (head) ctrl->t_start = globaltimer_ns();

    // the first rows of the trace held so far to global memory (one warp)
    auto flush_trace = [&](int l0, int rows) {
        for (int i = (int)lane; i < rows; i += 32) {
            const int l = l0 + i;
            LevelTrace tr;
            tr.level = l;
            tr.dir = 0;
            tr.frontier = cd_count(sh.trace[i][0]);
            tr.edges = cd_degree(sh.trace[i][0]);
            tr.t_ns = sh.trace[i][1];
            ctrl->trace[l < TRACE_CAP - 1 ? l : TRACE_CAP - 1] = tr;
        }
    };

    unsigned long long reached = 0, edges = 0;
    int roots = 0, L = 0;
    for (;; ++L) {
        const int par = L & 1;
        // 1. what all CTAs marked among this one's vertices; the other bitmap,
        // which every CTA has read before the last barrier, is cleared
        for (int i = t; i < (int)ctas * (W / 4); i += BLOCK) {
            const int w4 = i & (W / 4 - 1), c = i / (W / 4);
            const unsigned at = smem_addr(&sh.bits[par][rank * W + 4 * w4]);
            const uint4 x = alone ? *reinterpret_cast<const uint4 *>(&sh.bits[par][4 * w4])
                                  : remote_load_u4(map_rank(at, (unsigned)c));
            const unsigned m[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned nw = m[k] & ~sh.visited[4 * w4 + k];
                if (nw) atomicOr(&sh.fresh[4 * w4 + k], nw);
            }
            reinterpret_cast<uint4 *>(sh.bits[par ^ 1])[i] = make_uint4(0, 0, 0, 0);
        }
        if (t == 0) sh.rows[par ^ 1] = sh.longs[par ^ 1] = sh.verts[par ^ 1] = sh.degs[par ^ 1] = 0;
        __syncthreads();
        // 2. their rows (a word of fresh bits is one warp's alone)
        unsigned words = 0, verts = 0, degs = 0, shorts = 0, mine = 0;
        int b[PER], d[PER];
        unsigned m[PER];
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int v = i * BLOCK + t;
            const unsigned nw = sh.fresh[v >> 5];
            b[i] = d[i] = 0;
            if (nw >> lane & 1u) {
                sh.level[v] = L;
                b[i] = sh.row[v];
                d[i] = sh.row[v + 1] - b[i];
            }
            __syncwarp();  // every lane has read the word
            if (lane == (unsigned)i && nw) {
                sh.visited[v >> 5] |= nw;
                sh.fresh[v >> 5] = 0;
            }
            m[i] = __ballot_sync(FULL, d[i] > 0 && d[i] < SM_LONG);
            words |= nw;
            verts += __popc(nw);
            shorts += __popc(m[i]);
            mine += (unsigned)d[i];
        }
        if (words) {
            degs = __reduce_add_sync(FULL, mine);
            unsigned at = 0;
            if (lane == 0) {
                at = atomicAdd(&sh.rows[par], shorts);
                atomicAdd(&sh.verts[par], verts);
                atomicAdd(&sh.degs[par], degs);
            }
            at = __shfl_sync(FULL, at, 0);
#pragma unroll
            for (int i = 0; i < PER; i++) {
                if (m[i] >> lane & 1u) sh.list[at + __popc(m[i] & lanemask_lt())] = make_int2(b[i], b[i] + d[i]);
                at += __popc(m[i]);
                if (d[i] >= SM_LONG) sh.list[S - 1 - atomicAdd(&sh.longs[par], 1u)] = make_int2(b[i], b[i] + d[i]);
            }
        }
        __syncthreads();
        const int rows = (int)sh.rows[par], longs = (int)sh.longs[par];
        const unsigned long long cd_mine = cd_pack(sh.verts[par], sh.degs[par]);
        if (!alone && t < (int)ctas) remote_store_u64(map_rank(smem_addr(&sh.slot[par][rank]), (unsigned)t), cd_mine);
        // 3. the rows' neighbours
        unsigned *const next = sh.bits[par ^ 1];
        auto mark = [&](int w) {
            if (w < 0) return;
            const unsigned bit = 1u << (w & 31);
            if (!(next[w >> 5] & bit)) atomicOr(next + (w >> 5), bit);
        };
        for (int k = 0; k < longs; k++) {
            const int2 e = sh.list[S - 1 - k];
            for (int i = e.x + t; i < e.y; i += 4 * BLOCK) {
                int w[4];
#pragma unroll
                for (int q = 0; q < 4; q++) w[q] = i + q * BLOCK < e.y ? __ldg(a.col + i + q * BLOCK) : -1;
#pragma unroll
                for (int q = 0; q < 4; q++) mark(w[q]);
            }
        }
        const unsigned es = sh.degs[par] << skewed, rs = (unsigned)rows;
        const int lg = es <= 8 * rs ? 2 : es <= 16 * rs ? 3 : es <= 32 * rs ? 4 : 5, G = 1 << lg;
        const int sub = t & (G - 1), step = BLOCK >> lg;
        for (int r = t >> lg; r < rows; r += 2 * step) {
            const int2 e0 = sh.list[r], e1 = r + step < rows ? sh.list[r + step] : make_int2(0, 0);
            int i0 = e0.x + sub, i1 = e1.x + sub;
            while (i0 < e0.y || i1 < e1.y) {
                int w[4];
                w[0] = i0 < e0.y ? __ldg(a.col + i0) : -1;
                w[1] = i0 + G < e0.y ? __ldg(a.col + i0 + G) : -1;
                w[2] = i1 < e1.y ? __ldg(a.col + i1) : -1;
                w[3] = i1 + G < e1.y ? __ldg(a.col + i1 + G) : -1;
#pragma unroll
                for (int q = 0; q < 4; q++) mark(w[q]);
                i0 += 2 * G;
                i1 += 2 * G;
            }
        }
        unsigned long long cd = cd_mine;
        if (alone) {
            __syncthreads();
        } else {
            cluster_barrier();
            cd = 0;
            for (unsigned c = 0; c < ctas; c++) cd += sh.slot[par][c];
        }
        if (cd_count(cd) == 0) break;
        if (L == 0) roots = (int)cd_count(cd);
        reached += cd_count(cd);
        edges += cd_degree(cd);
        if (rank == 0 && warp == 0) {
            if (lane == 0) {
                sh.trace[L % SM_TRACE][0] = cd;
                sh.trace[L % SM_TRACE][1] = globaltimer_ns();
            }
            __syncwarp();
            if (L % SM_TRACE == SM_TRACE - 1) flush_trace(L - (SM_TRACE - 1), SM_TRACE);
            __syncwarp();
        }
    }
    for (int v = t; v < own; v += BLOCK) a.level[base + v] = sh.level[v];
    if (rank == 0 && warp == 0) flush_trace(L - L % SM_TRACE, L % SM_TRACE);
    if (head) {
        BfsOut o;
        o.levels = L;
        o.td_levels = L;
        o.bu_levels = 0;
        o.roots = roots;
        o.reached = reached;
        o.edges_c = edges;
        *a.out = o;
        ctrl->t_end = ctrl->t_exit = globaltimer_ns();
        ctrl->trace_len = L < TRACE_CAP ? L : TRACE_CAP;
        ctrl->rs.done = 1;
        ctrl->rs.mode = RESUME_LEVEL;
    }
}

// args null: whether the device holds the largest such cluster at all
// (cudaErrorInvalidConfiguration: no).
template <int LOGS, int BLOCK, typename RT>
cudaError_t small_launch(const BfsArgs *args, cudaStream_t st)
{
    static LaunchSetup setup;  // per template instance
    const size_t smem = sizeof(SmallShared<LOGS>);
    int unused = 0, fits = 0;
    auto config = [&](int c, cudaLaunchAttribute *at) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)c);
        cfg.blockDim = dim3(BLOCK);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = (unsigned)c;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cfg;
    };
    cudaError_t e = setup.get(unused, fits, [&](int, int &, int &fit_out) {
        auto *fn = k_bfs_small<LOGS, BLOCK, RT>;
        cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (r == cudaSuccess) r = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = config(SM_CTAS, &at);
        if (r == cudaSuccess) r = cudaOccupancyMaxActiveClusters(&fit_out, fn, &cfg);
        return r;
    });
    if (e != cudaSuccess) return e;
    if (fits < 1) return cudaErrorInvalidConfiguration;
    if (!args) return cudaSuccess;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = config((args->n + (1 << LOGS) - 1) >> LOGS, &at);
    return cudaLaunchKernelEx(&cfg, k_bfs_small<LOGS, BLOCK, RT>, *args);
}

template <typename RT>
cudaError_t small_launch_n(int n, const BfsArgs *a, cudaStream_t st)
{
    switch (small_part_log(n)) {
    case 10: return small_launch<10, 1024, RT>(a, st);
    case 11: return small_launch<11, 1024, RT>(a, st);
    case 12: return small_launch<12, 1024, RT>(a, st);
    default: return small_launch<SMALL_MAX_LOG, 1024, RT>(a, st);
    }
}

// (a device that has no room for the cluster, or whose set-up fails: the grid kernel)
bool small_fits(const DeviceCsr &g)
{
    const cudaError_t e = g.wide ? small_launch_n<long long>(g.n, nullptr, nullptr) : small_launch_n<int>(g.n, nullptr, nullptr);
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e == cudaSuccess;
}

}  // namespace

// Up to what the cluster's shared memory holds, and no graph of small degree
// (its long searches are the label-correcting kernel's).  Against the grid
// kernel (device us, cluster and grid):
//   top-down: uniform random, 65,536 vertices: 524 K edges 45 and 91, 2.1 M 56
//   and 75; 131,072 and 4.0 M: 92 and 104; RMAT, 65,536 and 3.4 M: 93 and 105.
//   direction-optimising, where the grid kernel's bottom-up steps skip most
//   edges of graphs that are dense or have hubs: uniform random, 65,536: 8
//   edges a vertex 45 and 75, 16: 46 and 67, 32: 56 and 50; 131,072, 15 a
//   vertex: 72 and 101; RMAT: 16,384 vertices, 426 K edges: 34 and 42; 32,768,
//   530 K: 41 and 49; 65,536: 381 K 46 and 48, 740 K 52 and 50.
// Nor a graph of which one CTA would walk too much, as every level is the time of
// its slowest CTA and the grid kernel deals rows to all SMs: the costliest part of
// small_row_cost, and the longest row.  (us here and in the grid kernel) top-down:
// uniform random, 16,000 vertices, 261 K entries in a part: 53 and 84, 517 K with
// rows of 512 among them: 174 and 127; 2,000, 820 K: 348 and 87; a clique of 1,000
// of 131,000 vertices: 408 and 96; a star of 20,000: 24 and 24, of 131,000: 90 and
// 27.  Direction-optimising: uniform random, 16,000 vertices, 66 K in a part: 31 and
// 37, 131 K 39 and 37; 131,072, 66 K: 66 and 70, 132 K 74 and 58; RMAT, 16,384
// vertices, a cost of some 73 K: 33 and 39, 117 K 43 and 38; 131,072, 80 K: 61 and
// 55; a star of 5,000: 14 and 19, of 20,000: 25 and 20.
bool bfs_small(const DeviceCsr &g, const gbfs_params &p)
{
    if (p.per_level_launch || p.direction == GBFS_DIR_BOTTOMUP || bfs_relax_tail(g, p)) return false;
    if (g.n > SMALL_MAX_N || g.m > 4 << 20 || g.max_degree > 1 << 14) return false;
    const int64_t most = p.direction == GBFS_DIR_TOPDOWN ? 250000 : g.n <= SMALL_MAX_N / 2 ? 100000 : 70000;
    if (g.part_cost > most) return false;
    if (p.direction != GBFS_DIR_TOPDOWN &&
        g.m > (small_skewed(g.max_degree, g.n, g.m) ? (int64_t)1 << 19 : 20 * (int64_t)g.n))
        return false;
    return small_fits(g);
}

cudaError_t bfs_small_launch(const BfsArgs &a, cudaStream_t st)
{
    return a.wide ? small_launch_n<long long>(a.n, &a, st) : small_launch_n<int>(a.n, &a, st);
}

}  // namespace gbfs
