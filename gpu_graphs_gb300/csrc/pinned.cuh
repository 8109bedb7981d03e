// pinned.cuh -- small pinned host blocks for results that kernels write.
//
// A pinned allocation costs about 100 us and its release 150, whatever its
// size, more than a search of a small graph.  Slots are carved from 64 KB slabs
// shared by the process (any thread, any device); a slab goes back once its
// slots have, except one that is kept.
#pragma once

#include <cstddef>

namespace gbfs {

constexpr size_t PINNED_SLOT = 512;

// A zeroed slot of PINNED_SLOT bytes, readable and writable by kernels at the
// same address; null when pinned memory has run out.
void *pinned_slot_take();
void pinned_slot_give(void *slot);

// A slot held by a scope, as a T (what a device -> host copy of a few words
// lands in: into pageable memory it takes 12 us).
template <typename T>
struct Pinned {
    static_assert(sizeof(T) <= PINNED_SLOT, "fits a slot");
    T *p;
    Pinned() : p((T *)pinned_slot_take()) {}
    ~Pinned() { pinned_slot_give(p); }
    Pinned(const Pinned &) = delete;
    Pinned &operator=(const Pinned &) = delete;
    explicit operator bool() const { return p != nullptr; }
    T *operator->() const { return p; }
};

}  // namespace gbfs
