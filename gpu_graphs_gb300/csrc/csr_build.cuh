// csr_build.cuh -- on-device edge list -> CSR builder.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace gbfs {

// A CSR resident in HBM.  Rows of graphs built from edges are sorted
// ascending.  zmask bit v is set when out-degree(v) == 0.
struct DeviceCsr {
    // one allocation for the arrays of a vertex's size: zmask, heavy, first and
    // second, and the row offsets of a graph built here (a given CSR's are its own)
    void *block = nullptr;
    bool own_row = false;      // row / row64 is an allocation of its own
    // a few bytes: the driver maps memory for small allocations 2 MB at a time and
    // unmaps it with the last of them, some 100 us each way, which calls that only
    // use a little scratch would pay again and again (another graph taken over
    // beside this one: 380 us without it, 270 so)
    void *keep = nullptr;
    int32_t n = 0;
    int64_t m = 0;
    int *row = nullptr;        // n+1 (null when wide)
    long long *row64 = nullptr;  // n+1, wide graphs only: 64-bit row offsets (more than 2^31-1 edges)
    bool wide = false;
    int *col = nullptr;        // m
    unsigned *zmask = nullptr; // (n+31)/32
    int32_t max_degree = 0;
    int64_t nonisolated = 0;
    int64_t part_cost = 0;     // graphs of up to SMALL_MAX_N vertices: largest sum of small_row_cost in a part
    int *heavy = nullptr;      // vertices of out-degree > HEAVY_DEGREE (any order)
    int32_t nheavy = 0;
    // each row's first and second entries, -1 where the row is shorter (with
    // hub-first rows, the first is the highest-degree neighbour): bottom-up's
    // first probe, read coalesced
    int *first = nullptr;      // n
    int *second = nullptr;     // n; not allocated for hub-first rows (probed at the first entry alone)
    bool hub_rows = false;     // rows are hub-first (csr_hub_first ran)
    bool sorted_rows = false;  // every row is known to be ascending
    // fixed-width adjacency of a small-degree graph, built on demand by
    // csr_build_quads for the label-correcting kernel: quad[v] holds row v's
    // entries, -1 past its end; a row of more than four keeps its first three
    // there and a link -2 - k in the fourth place to its node, over[16 k ..]:
    // the entries from the fourth on (-1 past the end) and, last, its degree
    int32_t nover4 = 0;        // rows of more than four entries
    int4 *quad = nullptr;      // n; the allocation of both
    int *over = nullptr;       // 16 per row of more than four entries
    // multi-source pull pieces (built on demand by ms_prepare): every row of
    // degree > 2 * MS_PIECE contributes {vertex, j} for its j-th MS_PIECE edges
    int2 *pieces = nullptr;
    int32_t npieces = 0;
    int64_t pieces_bytes = 0;  // of pieces and tpieces together
    bool pieces_built = false;
    // transpose (in-edges), built on demand for bottom-up steps on graphs
    // whose in-edges differ from their out-edges; rows unsorted
    int *trow = nullptr;       // n+1
    int *tcol = nullptr;       // m
    int *tfirst = nullptr;     // n: the transpose's first entries (its rows are hub-first)
    int *theavy = nullptr;     // vertices of in-degree > HEAVY_DEGREE (built with the transpose)
    int32_t ntheavy = 0;
    // multi-source pull pieces over the transpose (ms_prepare, once trow exists)
    int2 *tpieces = nullptr;
    int32_t ntpieces = 0;
    bool tpieces_built = false;
};

// Graphs that one thread-block cluster may search (bfs_small.cu): the cluster's
// CTAs own aligned parts of 2^small_part_log vertices each.
constexpr int SMALL_CTAS = 16;
constexpr int SMALL_MAX_LOG = 13;
constexpr int SMALL_MAX_N = SMALL_CTAS << SMALL_MAX_LOG;
constexpr int SMALL_LONG = 512;  // rows that the whole CTA walks, one after another

inline int small_part_log(int32_t n)
{
    int l = 10;
    while (SMALL_CTAS << l < n) l++;
    return l;
}

// What walking a row of d entries costs a CTA there, in entries of short rows
// (about 0.1 ns): a long row is a step of its own (0.35 us), and has more
// neighbours per word to mark.
__host__ __device__ inline long long small_row_cost(int d)
{
    if (d < SMALL_LONG) return d;
    return 3ll * d > 3500 ? 3ll * d : 3500;
}

// Rows longer than this are walked by a whole warp in multi-source passes.
constexpr int HEAVY_DEGREE = 64;

// Build from device edge arrays (m entries each).  Returns a GBFS_* status;
// on failure `err` says why.  All work is ordered on `st`; the call
// synchronises `st` before returning.  The row offsets are 64-bit (`wide`)
// when the edges to store could exceed 2^31-1, or with GBFS_WIDE_ROWS.
int csr_build_from_edges(int32_t n, int64_t m, const int *d_src, const int *d_dst,
                         unsigned flags, cudaStream_t st, DeviceCsr &out, std::string &err);

// The ways this thread's last csr_build_from_edges took (for tests).
enum BuildRoute : int {
    BUILD_BUCKETS = 1,    // entries by buckets of rows
    BUILD_LONG_BITS = 2,  // rows of more than 4,096 entries through bitmaps
    BUILD_4K_BITS = 4,    // rows of 2,049 to 4,096 entries too
};
int csr_build_route();

// Take an existing device CSR (row n+1, col m; ownership moves to `out`),
// validate it and compute zmask / max_degree / nonisolated.
int csr_adopt(int32_t n, int64_t m, int *d_row, int *d_col, cudaStream_t st, DeviceCsr &out,
              std::string &err);
// The same with 64-bit row offsets (a wide graph).
int csr_adopt64(int32_t n, int64_t m, long long *d_row, int *d_col, cudaStream_t st, DeviceCsr &out,
                std::string &err);

// in-edges == out-edges?  Rows need not be sorted (a sorted copy is checked);
// c.sorted_rows is set from what the check finds.
int csr_check_symmetric(DeviceCsr &c, cudaStream_t st, bool &sym, std::string &err);

// Move each row's highest-degree neighbour to the row's front.
int csr_hub_first(DeviceCsr &c, cudaStream_t st, std::string &err);

// Build c.trow / c.tcol (the in-edge CSR, rows hub-first) with c.tfirst and
// c.theavy; a no-op once built.  Synchronises st.  Not for wide graphs
// (GBFS_ERR_TOO_LARGE: their searches stay top-down).
int csr_build_transpose(DeviceCsr &c, cudaStream_t st, std::string &err);

// (Re)compute c.first / c.second from the rows as they are now.  Synchronises st.
int csr_build_first(DeviceCsr &c, cudaStream_t st, std::string &err);

// Build c.quad / c.over; a no-op once built.  Only for graphs of out-degree at
// most QUAD_MAX_DEGREE.  Enqueued on st; no sync (work on other streams has to
// wait for it).
constexpr int QUAD_MAX_DEGREE = 16;
int csr_build_quads(DeviceCsr &c, cudaStream_t st, std::string &err);
// Bytes csr_build_quads allocates.
int64_t csr_quad_bytes(const DeviceCsr &c);
void csr_drop_quads(DeviceCsr &c);

// Device bytes held by the CSR and everything built on it.
int64_t csr_device_bytes(const DeviceCsr &c);

void csr_free(DeviceCsr &c);

}  // namespace gbfs
