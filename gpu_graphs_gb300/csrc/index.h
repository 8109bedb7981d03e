// index.h -- entry indices up to the largest of their type (host and device).
//
// A graph with 32-bit row offsets may hold 2^31 - 1 entries, so the sums that a
// loop forms past the end of its range (the next step, the next lane) need not
// fit the type.
#pragma once

#ifdef __CUDACC__
#define GBFS_HD __host__ __device__ __forceinline__
#else
#define GBFS_HD inline
#endif

namespace gbfs {

// Thread t's part of the entries [s, e), BLOCK threads wide and ILP at a time:
// v = load(i) of each entry i, then use(v, true), and use(0, false) past the end,
// so that all threads make the same calls of use.
template <int BLOCK, int ILP, typename Load, typename Use>
GBFS_HD void walk_range(int s, int e, int t, Load load, Use use)
{
    const int len = e - s;
    for (int i0 = 0; i0 < len; i0 += ILP * BLOCK) {
        unsigned v[ILP];
#pragma unroll
        for (int q = 0; q < ILP; q++) v[q] = i0 + q * BLOCK + t < len ? load(s + (i0 + q * BLOCK + t)) : 0u;
#pragma unroll
        for (int q = 0; q < ILP; q++) use(v[q], i0 + q * BLOCK + t < len);
    }
}

}  // namespace gbfs
