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

// i + k, which may lie past the type's largest value: then it is before no end.
template <typename T>
GBFS_HD T idx_add(T i, int k)
{
    if constexpr (sizeof(T) == sizeof(int)) return (T)((unsigned)i + (unsigned)k);
    else return i + k;
}

// i < e for an entry index i from idx_add and a range's end e (less than 2^31 apart).
template <typename T>
GBFS_HD bool idx_before(T i, T e)
{
    if constexpr (sizeof(T) == sizeof(int)) return (int)((unsigned)e - (unsigned)i) > 0;
    else return i < e;
}

// min(i + k, e)
template <typename T>
GBFS_HD T idx_end(T i, int k, T e)
{
    const T x = idx_add(i, k);
    return idx_before(x, e) ? x : e;
}

// (lo + hi) / 2 for 0 <= lo <= hi
template <typename T>
GBFS_HD T idx_mid(T lo, T hi)
{
    return lo + (hi - lo) / 2;
}

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
