// tile_common.cuh -- what the two leaf-pair tile kernels share (tiles.cu: every class and
// geometry, one pair per lane and step; tile_packed.cu: the common ones, two pairs per lane
// and step).
#pragma once

#include <cstdint>

#include "tc_internal.cuh"
#include "traverse2pt.hpp"
#include "pair_math.cuh"

namespace tc {

enum { TG_FLAT = 0, TG_ARC = 1, TG_SPHEUC = 2, TG_3D = 3 };   // geometry
enum { TK_NN = 0, TK_SC = 1, TK_GEN = 2, TK_GG = 3 };           // class family

__host__ __device__ inline size_t bins_bytes(int nq, int nb)
{
    return ((size_t)nq * nb * 8 + (size_t)nb * 8 + (size_t)nq * nb * 4 + 15) & ~(size_t)15;
}

__host__ __device__ inline size_t edges_bytes(int nb)
{
    return ((size_t)2 * (nb + 1) * 4 + 15) & ~(size_t)15;
}

__device__ __forceinline__ float warp_max(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sums v[0..7] over the warp: after the reduce-scatter each group of 4 lanes holds one value's
// total; lane 4 q + 0 returns value q's total in *out (q = 0..7) and true.
__device__ __forceinline__ bool warp_sum8(float (&v)[8], int lane, float& out)
{
    // xor 16: keep 4 of 8.
    const bool h16 = lane & 16;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float send = h16 ? v[q] : v[q + 4];
        const float got = __shfl_xor_sync(0xffffffffu, send, 16);
        v[q] = (h16 ? v[q + 4] : v[q]) + got;
    }
    // xor 8: keep 2 of 4.
    const bool h8 = lane & 8;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float send = h8 ? v[q] : v[q + 2];
        const float got = __shfl_xor_sync(0xffffffffu, send, 8);
        v[q] = (h8 ? v[q + 2] : v[q]) + got;
    }
    // xor 4: keep 1 of 2.
    const bool h4 = lane & 4;
    {
        const float send = h4 ? v[0] : v[1];
        const float got = __shfl_xor_sync(0xffffffffu, send, 4);
        v[0] = (h4 ? v[1] : v[0]) + got;
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    out = v[0];
    return (lane & 3) == 0;
}

// Which value a lane holds after warp_sum8: bit 4 picks the upper half, bit 3 the upper
// quarter of that, bit 2 the upper one of the last two.
__device__ __forceinline__ int warp_sum8_index(int lane)
{
    return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}

// A leaf pair decided in FP64 with the reference's formulas: decide64 (the reference's
// process11 for s1 = s2 = 0) on the FP64 leaf positions.  Out of line: it runs for about one
// pair in 10^5, and keeping it out of the loop keeps the loop's registers low.
static __device__ __noinline__ int leaf_pair64(const TravParams& T, int ida, int idb, bool self,
                                        float* r, float* logr)
{
    const double* x2 = self ? T.x1 : T.x2;
    const double* y2 = self ? T.y1 : T.y2;
    const double* z2 = self ? T.z1 : T.z2;
    const double dx = T.x1[ida] - x2[idb], dy = T.y1[ida] - y2[idb];
    double dsq = dx * dx + dy * dy;
    if (T.coords != FLAT) {
        const double dz = T.z1[ida] - z2[idb];
        dsq += dz * dz;
    }
    const Decision D = decide64(T, dsq, 0., 0.);
    if (D.act != ACT_ACCEPT) return -1;
    *r = D.r;
    *logr = D.logr;
    return D.k;
}

// The great-circle angle from a chord c < 0.25 (the tile checks it): the Maclaurin series
// of 2 asin(c / 2) to x^7, x = c / 2 (the first omitted term is below 2e-9 of x).
__device__ __forceinline__ float arc_series(float c)
{
    const float x = 0.5f * c, x2 = x * x;
    return 2.f * x * fmaf(x2, fmaf(x2, fmaf(x2, 5.f / 112.f, 3.f / 40.f), 1.f / 6.f), 1.f);
}

// Adds a tile's per-lane sums of one bin into the warp's FP32 bins.  acc: weight, sum w w r,
// sum w w lr (lr = log2(r^2 / edge^2) of the tile's reference edge), products; the bin's
// meanlogr sum is (ln 2 / 2) sum w w lr + log(edge) sum w w.
__device__ __forceinline__ void tile_bin_out(float (&acc)[8], unsigned cn, int kb, int nq, int nb,
                                             float ledge, float* fb, unsigned long long* np,
                                             bool quick, bool single, int lane)
{
    if (!__any_sync(0xffffffffu, cn != 0u) || kb >= nb) return;
    acc[2] = fmaf(acc[2], 0.5f * 0.69314718f, acc[0] * ledge);
    float tot;
    const bool holder = warp_sum8(acc, lane, tot);
    const int q = warp_sum8_index(lane);
    if (holder && q < nq) fb[q * nb + kb] += tot;
    if (!quick) {
        if (single) {
            const unsigned ct = __reduce_add_sync(0xffffffffu, cn);
            if (lane == 0) np[kb] += ct;
        } else if (cn) {
            atomicAdd(&np[kb], (unsigned long long)cn);
        }
    }
    __syncwarp();
}

// Adds the pairs that lanes hold for the shared bins (kx >= 0, values v) in ascending lane
// order: lane q < nq adds quantity q of each, so the sums do not depend on the order in which
// conflicting shared atomics would land.
__device__ __forceinline__ void shared_bins_in_order(int kx, const float (&v)[8], float* fb,
                                                     int nq, int nb, int lane)
{
    unsigned m = __ballot_sync(0xffffffffu, kx >= 0);
    while (m) {
        const int t = __ffs(m) - 1;
        m &= m - 1u;
        const int kt = __shfl_sync(0xffffffffu, kx, t);
        float x = 0.f;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const float y = __shfl_sync(0xffffffffu, v[q], t);
            x = lane == q ? y : x;
        }
        if (lane < nq) fb[lane * nb + kt] += x;
    }
}

}  // namespace tc
