// roots.cuh -- the top-level work items of a traversal, generated on the fly from an index
// (BaseCorr2::process, src/Corr2.cpp:146-288), shared by the breadth-first expansion and the
// depth-first walk.
#pragma once

#include <cstdint>

#include "tc_internal.cuh"
#include "traverse2pt.hpp"

namespace tc {

// Row i of the upper triangle (self + pairs j > i) of n top cells starts at
// i*n - i*(i-1)/2; item g of that enumeration.  The row is the floor of the root of a
// quadratic whose discriminant is exact in 64 bits; an FP32 square root of it is off by a
// fraction of a row (a few rows for n above 2^23), which the two loops put right.
__device__ __forceinline__ void tri_index(long long n, long long g, long long& i, long long& j)
{
    const long long b = 2 * n + 1;
    i = (long long)(((float)b - sqrtf((float)(b * b - 8 * g))) * 0.5f);
    if (i < 0) i = 0;
    if (i > n - 1) i = n - 1;
    while (i > 0 && i * n - i * (i - 1) / 2 > g) --i;
    while (i + 1 < n && (i + 1) * n - (i + 1) * i / 2 <= g) ++i;
    j = g - (i * n - i * (i - 1) / 2) + i;
}

// g / n and g % n; in 32 bits where both fit, a quarter of the instructions.
__device__ __forceinline__ void div_index(long long n, long long g, long long& i, long long& j)
{
    if ((unsigned long long)(g | n) >> 32) { i = g / n; j = g - i * n; return; }
    const unsigned q = (unsigned)g / (unsigned)n;
    i = q;
    j = (unsigned)g - q * (unsigned)n;
}

// Item r of the roots of patch pair p.
__device__ __forceinline__ int2 make_pair_root(const TravParams& T, int p, long long r)
{
    const int2 pr = T.ppairs[p];
    const int* ti = T.ptop + T.ptop_off[pr.x];
    long long i, j;
    if (pr.x == pr.y) {
        tri_index(T.ptop_off[pr.x + 1] - T.ptop_off[pr.x], r, i, j);
        return j == i ? make_int2(ti[i], -1) : make_int2(ti[i], ti[j]);
    }
    div_index(T.ptop_off[pr.y + 1] - T.ptop_off[pr.y], r, i, j);
    return make_int2(ti[i], T.ptop[T.ptop_off[pr.y] + j]);
}

// Patches: root g of all patch pairs (auto enumeration within a patch, all top pairs
// across two patches).
__device__ __forceinline__ int2 make_patch_root(const TravParams& T, long long g)
{
    int lo = 0, hi = T.npair;          // proot_off[lo] <= g < proot_off[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (T.proot_off[mid] <= g) lo = mid; else hi = mid;
    }
    return make_pair_root(T, lo, g - T.proot_off[lo]);
}

template <int MODE = 0>
__device__ __forceinline__ int2 make_root(const TravParams& T, long long g)
{
    if constexpr (MODE == 3) return make_patch_root(T, g);
    if (g >= T.ngen) return T.in_tasks[g - T.ngen];
    long long i, j;
    if (T.autoc) {
        tri_index(T.ntop1, g, i, j);
        return j == i ? make_int2(T.tops1[i], -1) : make_int2(T.tops1[i], T.tops1[j]);
    }
    div_index(T.ntop2, g, i, j);
    return make_int2(T.tops1[i], T.tops2[j]);
}

}  // namespace tc
