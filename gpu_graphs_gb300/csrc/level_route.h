// level_route.h -- how a batch's levels reach an output (host only).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <utility>
#include <vector>

namespace gbfs {

enum class LevelRoute {
    KERNEL,  // stored by k_slices_out
    COPY,    // a device copy: memory of another GPU, which a kernel may not reach
    HOST,    // through the pinned staging of the union's levels
};

// type: cudaMemoryType of the output (0: unregistered, 1: host, 2: device, 3:
// managed), ptr_device: the GPU its memory is on, device: the graph's GPU.  An
// output that is not aligned for a kernel's stores is copied as well.
inline LevelRoute level_route(const void *p, int type, int ptr_device, int device)
{
    if (type != 2 && type != 3) return LevelRoute::HOST;
    if (reinterpret_cast<uintptr_t>(p) % alignof(int32_t) != 0) return LevelRoute::COPY;
    return type == 3 || ptr_device == device ? LevelRoute::KERNEL : LevelRoute::COPY;
}

// Whether two of the device outputs [out[i], out[i] + count[i]) overlap: then they
// are all copied, in order, so that the last one stands.
// (Outputs in ascending order, as slices of one array are, take one pass; others
// are sorted, in `scratch`, which may throw std::bad_alloc.)
inline bool outputs_overlap(const int32_t *const *out, const int32_t *count, const LevelRoute *route, size_t n,
                            std::vector<std::pair<uintptr_t, uintptr_t>> &scratch)
{
    auto range = [&](size_t i) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(out[i]);
        return std::make_pair(b, b + sizeof(int32_t) * (size_t)count[i]);
    };
    uintptr_t end = 0;
    bool ascending = true;
    for (size_t i = 0; i < n && ascending; i++) {
        if (route[i] == LevelRoute::HOST) continue;
        const auto r = range(i);
        ascending = r.first >= end;
        end = r.second;
    }
    if (ascending) return false;
    scratch.clear();
    for (size_t i = 0; i < n; i++)
        if (route[i] != LevelRoute::HOST) scratch.push_back(range(i));
    std::sort(scratch.begin(), scratch.end());
    for (size_t i = 1; i < scratch.size(); i++)
        if (scratch[i].first < scratch[i - 1].second) return true;
    return false;
}

}  // namespace gbfs
