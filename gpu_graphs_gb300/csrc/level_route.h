// level_route.h -- how a batch's levels reach an output (host only).
#pragma once

namespace gbfs {

enum class LevelRoute {
    KERNEL,  // stored by k_slices_out
    COPY,    // a device copy: memory of another GPU, which a kernel may not reach
    HOST,    // through the pinned staging of the union's levels
};

// type: cudaMemoryType of the output (0: unregistered, 1: host, 2: device, 3:
// managed), ptr_device: the GPU its memory is on, device: the graph's GPU.
inline LevelRoute level_route(int type, int ptr_device, int device)
{
    if (type == 3) return LevelRoute::KERNEL;
    if (type != 2) return LevelRoute::HOST;
    return ptr_device == device ? LevelRoute::KERNEL : LevelRoute::COPY;
}

}  // namespace gbfs
