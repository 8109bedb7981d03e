// parents.cuh -- canonical BFS-tree parents from a level array.
#pragma once

#include <cuda_runtime.h>

#include "csr_build.cuh"

namespace gbfs {

struct BfsCtrl;

// parent[v] = smallest u with an edge u -> v and level[u] == level[v] - 1;
// -1 for level <= 0 (the source, unreached).  d_level must be a complete BFS
// level array of g from `source`.  Rows longer than MS_HUGE are split over the
// GPU where g's pieces have been built (ms_prepare).  ctrl: of the search that
// wrote d_level, for its trace (null: none).  Enqueued on st; no sync.
cudaError_t parents_enqueue(const DeviceCsr &g, bool symmetric, int source, const int *d_level, const BfsCtrl *ctrl,
                            int *d_parent, cudaStream_t st);

}  // namespace gbfs
