// pinned.cu -- see pinned.cuh.
#include "pinned.cuh"

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

namespace gbfs {

namespace {

constexpr int SLOTS = 128;

struct Slab {
    char *mem = nullptr;
    int used = 0;
    bool taken[SLOTS] = {};
};

std::mutex g_mu;
std::vector<Slab> g_slabs;

}  // namespace

void *pinned_slot_take()
{
    std::lock_guard<std::mutex> lk(g_mu);
    Slab *s = nullptr;
    for (auto &x : g_slabs)
        if (x.used < SLOTS) s = &x;
    if (!s) {
        Slab fresh;
        if (cudaHostAlloc((void **)&fresh.mem, SLOTS * PINNED_SLOT, cudaHostAllocPortable | cudaHostAllocMapped) !=
            cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        try {
            g_slabs.push_back(fresh);
        } catch (const std::bad_alloc &) {
            cudaFreeHost(fresh.mem);
            return nullptr;
        }
        s = &g_slabs.back();
    }
    int i = 0;
    while (s->taken[i]) i++;
    s->taken[i] = true;
    s->used++;
    char *p = s->mem + i * PINNED_SLOT;
    memset(p, 0, PINNED_SLOT);
    return p;
}

void pinned_slot_give(void *slot)
{
    if (!slot) return;
    std::lock_guard<std::mutex> lk(g_mu);
    size_t at = g_slabs.size();
    int empty = 0;
    for (size_t k = 0; k < g_slabs.size(); k++) {
        Slab &x = g_slabs[k];
        if ((char *)slot >= x.mem && (char *)slot < x.mem + SLOTS * PINNED_SLOT) {
            x.taken[((char *)slot - x.mem) / PINNED_SLOT] = false;
            x.used--;
            at = k;
        }
        empty += x.used == 0;
    }
    if (at < g_slabs.size() && g_slabs[at].used == 0 && empty > 1) {
        cudaFreeHost(g_slabs[at].mem);
        g_slabs.erase(g_slabs.begin() + (long)at);
    }
}

}  // namespace gbfs
