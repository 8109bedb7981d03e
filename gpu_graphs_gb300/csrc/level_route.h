// level_route.h -- how a batch's levels reach an output (host only).
#pragma once

#include <cstdint>

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

}  // namespace gbfs
