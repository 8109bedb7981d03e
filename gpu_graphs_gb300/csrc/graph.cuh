// graph.cuh -- the opaque handle types behind the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "bfs.cuh"
#include "csr_build.cuh"
#include "msbfs.cuh"
#include "retry.h"

struct gbfs_graphset;

namespace gbfs {

// Servers and a graph's fixed-width adjacency (csr.quad).  Counts go up under the
// graph's mutex, and the adjacency is freed under it, only while users is 0.
struct QuadHold {
    std::atomic<int> users{0};   // servers that serve the graph from it, in their budgets
    std::atomic<int> barred{0};  // servers whose budget has no room for it: it is not built
};

}  // namespace gbfs

struct gbfs_graph {
    gbfs::DeviceCsr csr;
    std::shared_ptr<gbfs::QuadHold> quads = std::make_shared<gbfs::QuadHold>();
    gbfs_params params{};        // read and written only under pmu (graph_params / set)
    mutable std::mutex pmu;
    gbfs::BfsWork work;
    gbfs::MsWork ms;
    cudaStream_t stream = nullptr;
    int device = 0;
    bool symmetric = false;      // in-edges == out-edges (bottom-up allowed)
    bool last_multi = false;     // the last traversal was multi-source (trace source)
    std::mutex mu;
    gbfs::Retry quad_retry, piece_retry;  // under mu
    // graph set cached by gbfs_bfs_batch_graphs (keyed by the handle list)
    std::vector<const gbfs_graph *> batch_key;
    gbfs_graphset *batch_set = nullptr;
};

struct gbfs_graphset {
    gbfs_graph *g = nullptr;           // the disjoint union
    std::vector<int64_t> offsets;      // count+1 vertex offsets
    std::vector<int32_t> sizes;        // n of each member
    // per member, where its levels go and start in the union (batch.cu); on
    // the device, allocated by the first call with device outputs
    struct Slice {
        int32_t *dst;
        long long offset;
    };
    Slice *d_slices = nullptr;
};

namespace gbfs {

// A copy of the graph's traversal parameters (other threads may set them).
inline gbfs_params graph_params(const gbfs_graph *g)
{
    std::lock_guard<std::mutex> lk(g->pmu);
    return g->params;
}

inline void graph_set_params(gbfs_graph *g, const gbfs_params &p)
{
    std::lock_guard<std::mutex> lk(g->pmu);
    g->params = p;
}

// thread-local error detail
void set_error(const std::string &msg);
int fail(int code, const std::string &msg);
bool is_device_ptr(const void *p);
int cuda_fail(cudaError_t e, const char *what);

// Make a handle around a built CSR (takes ownership of csr).
int graph_wrap(DeviceCsr &csr, bool symmetric_known, bool symmetric, cudaStream_t st,
               gbfs_graph **out);

}  // namespace gbfs
