// multipole.cu -- 3-point correlations with LogMultipole binning on sm_103a (all N / K / G
// classes: GGG's contraction over the payloads each class needs, see MPParams).
//
// Semantics follow the reference's multipole algorithm (Porth et al.):
//   BaseCorr3::multipole (src/Corr3.cpp:1124-1175; cross12 1177-1237; three-field
//   1239-1305), multipoleSplit1 (1374-1449), splitC2Cells (1323-1372), multipoleFinish
//   (1548-1679), splitC2CellsOrCalculateGn (1452-1546), Corr3::calculateGn +
//   MultipoleScratch<GData>::calculateGn (1681-1704, 1767-1828), Corr3::calculateZeta
//   (1861-2087) and MultipoleHelper<1..6>::CalculateZeta (2108-3082); scratch layout
//   include/MultipoleScratch.h:36-125, 296-383.
//
// GB300 design:
//   * Phase 1: one block per top-level cell walks the c1 subtree of multipoleSplit1, refining
//     the c2 list with block-parallel decisions and a stable block scan, and emits one job
//     (c1, c2 list) per cell that is small enough to start multipoleFinish.
//   * Phase 2: persistent blocks take jobs from a counter.  A job runs multipoleFinish as a
//     depth-first loop: each pass over the c2 list is block-parallel; every accepted pair
//     becomes a record of its FP64-computed terms stored as FP32 (phase z, projected shear,
//     scalar sums).  The records are ranked stably by bin and split evenly over the warps;
//     a warp forms z^n for n = 1..max_n+1 with one multiplicative warp scan per record, sums
//     the G_n / W_n terms in FP32 and flushes them to the FP64 scratch.  When c1 must split,
//     the scratch is copied into a free slot and the right child is pushed, as the
//     reference's mp.duplicate() does.
//   * Rows of Zeta that are final become vertex records (FP32 copies of G_n and W_n).  The
//     contraction over vertices is a sum of outer products per n; k_mp_zeta (zeta.cu) runs it
//     in batches (waves) between runs of the finish kernel, FP32 products with FP64 sums.
//   * A last kernel sums what was contracted in place, the contraction's sums and the diagonal
//     self-pair corrections in a fixed order.
//   * A three-field cross keeps vertex 3's pairs in scratch bins [nbd, 2 nbd), so the same
//     kernels produce both cross blocks of a (2 nbd)^2 matrix (MPParams::three).
// Geometry and the split/accept decisions are taken in FP32 with error margins
// (mp_decide32); an entry inside a margin is decided again in FP64 with the reference's
// arithmetic, so the decisions are the reference's.  The cell payloads are the tree's float
// values.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "tc_internal.cuh"
#include "tc_host.hpp"
#include "multipole.hpp"

namespace tc {

static constexpr int MB = 128;            // threads per multipole block
static constexpr int MBLK = 5;            // multipole blocks per SM (96 registers): 221 ms for the call
                                          // at k_mp_finish, 4: 232, 6: 289 (spills)
static constexpr int MW = MB / 32;        // warps per block
static constexpr int MSTACK = 128;        // depth of the block-local stacks

// ---------------------------------------------------------------------------------------
// Leaf sums of every cell: calculateSumWSq, calculateSumWZSq, calculateSumAbsWZSq
// (src/Cell.cpp:138-168).  A cell is a leaf of these sums if its size is 0, it holds one
// point, or it has no children; each such leaf adds w^2, (wz)^2 and |wz|^2 to itself and
// to every ancestor.

__global__ void k_leaf_sums(int ncap, Cells C, double* ls)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncap) return;
    if (C.n[i] <= 0) return;   // unused id
    const bool leaf = (C.size[i] == 0.f) || (C.n[i] == 1) || (C.left[i] < 0);
    if (!leaf) return;
    // Skip cells nested below another summation leaf (their sum is already counted there).
    for (int p = C.parent[i]; p >= 0; p = C.parent[p])
        if (C.size[p] == 0.f) return;
    const double w = C.w[i];
    const double gr = C.d1[i], gi = C.d2[i];
    const double v0 = w * w, v1 = gr * gr - gi * gi, v2 = 2. * gr * gi, v3 = gr * gr + gi * gi;
    for (int p = i; p >= 0; p = C.parent[p]) {
        atomicAdd(&ls[4 * (size_t)p + 0], v0);
        atomicAdd(&ls[4 * (size_t)p + 1], v1);
        atomicAdd(&ls[4 * (size_t)p + 2], v2);
        atomicAdd(&ls[4 * (size_t)p + 3], v3);
    }
}

__global__ void k_leaf_sums_f(int ncap, const double* ls, float4* lsf)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncap) return;
    const double* p = ls + 4 * (size_t)i;
    lsf[i] = make_float4((float)p[0], (float)p[1], (float)p[2], (float)p[3]);
}

// The cells of an N or K pair field as a real payload (GNN, GKK, NKK, KNN, KKK;
// MultipoleHelper<4> and <1>, src/Corr3.cpp:2462-2580, 2108-2214): (d1, d2) := (w, 0) for N
// (Sigma w z^n is its G_n), (w k, 0) for K; the leaf sums (sum w^2 or sum (w k)^2, 0) stand
// where the squared shear was.
__global__ void k_mp_scalar_pairs(int ncap, int is_n, TCell* tc, float* d1, float* d2,
                                  double* ls, float4* lsf)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncap) return;
    TCell c = tc[i];
    if (is_n) c.c.x = c.b.w;
    c.c.y = 0.f;
    tc[i] = c;
    d1[i] = c.c.x;
    d2[i] = 0.f;
    double* l = ls + 4 * (size_t)i;
    if (is_n) l[1] = l[0];
    l[2] = 0.;
    lsf[i] = make_float4((float)l[0], (float)l[1], 0.f, (float)l[3]);
}

int launch_scalar_pairs(int ncap, int is_n, TCell* tc, float* d1, float* d2, double* ls,
                        float4* lsf, cudaStream_t st)
{
    if (ncap <= 0) return 0;
    count_launch();
    k_mp_scalar_pairs<<<(ncap + 255) / 256, 256, 0, st>>>(ncap, is_n, tc, d1, d2, ls, lsf);
    TC_CU(cudaGetLastError());
    return 0;
}

int launch_leaf_sums(int ncap, const Cells& C, double* ls, float4* lsf, cudaStream_t st)
{
    TC_CU(cudaMemsetAsync(ls, 0, 4 * sizeof(double) * (size_t)ncap, st));
    count_launch();
    k_leaf_sums<<<(ncap + 255) / 256, 256, 0, st>>>(ncap, C, ls);
    TC_CU(cudaGetLastError());
    count_launch();
    k_leaf_sums_f<<<(ncap + 255) / 256, 256, 0, st>>>(ncap, ls, lsf);
    TC_CU(cudaGetLastError());
    return 0;
}

// ---------------------------------------------------------------------------------------
// FP64 geometry and rules.

struct C2 { double re, im; };
__device__ __forceinline__ C2 cmul(C2 a, C2 b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ C2 conj2(C2 a) { return {a.re, -a.im}; }
__device__ __forceinline__ C2 cadd(C2 a, C2 b) { return {a.re + b.re, a.im + b.im}; }

__device__ __forceinline__ void norm3(double& x, double& y, double& z)
{
    double n = sqrt(x * x + y * y + z * z);
    if (n == 0.) { x = 1.; y = 0.; z = 0.; } else { x /= n; y /= n; z /= n; }
}

__device__ __forceinline__ double mp_dist_sq(const MPParams& P, int i, int j)
{
    double dx = P.x[i] - P.x[j], dy = P.y[i] - P.y[j];
    if (P.coords == FLAT) return dx * dx + dy * dy;
    double dz = P.z[i] - P.z[j];
    double dsq = dx * dx + dy * dy + dz * dz;
    if (P.metric == ARC) { double th = 2. * asin(sqrt(dsq) / 2.); return th * th; }
    return dsq;
}

// BinTypeHelper<Log>::singleBin, include/BinType.h:93-151.
__device__ __forceinline__ bool mp_single_bin(const MPParams& P, double rsq, double s1ps2, int& ik,
                                              double& r, double& logr)
{
    if (s1ps2 == 0.) return true;
    double s2 = s1ps2 * s1ps2;
    if (s2 > P.asq * rsq) return false;
    if (s2 <= P.bsq * rsq) return true;
    if (s2 > 0.25 * (P.binsize + P.b) * (P.binsize + P.b) * rsq) return false;
    logr = 0.5 * log(rsq);
    double kk = (logr - P.logminsep) / P.binsize;
    ik = int(kk);
    double frac = kk - ik;
    double f = fmin(frac, 1. - frac);
    double t4 = f * P.binsize + P.b;
    if (s2 > t4 * t4 * rsq) return false;
    double t5 = frac * P.binsize + P.b - s2 / rsq;
    if (s2 > t5 * t5 * rsq) return false;
    r = sqrt(rsq);
    return true;
}

__device__ __forceinline__ bool mp_too_small(const MPParams& P, double rsq, double s)
{ return rsq < P.minsepsq && s < P.minsep && rsq < (P.minsep - s) * (P.minsep - s); }
__device__ __forceinline__ bool mp_too_large(const MPParams& P, double rsq, double s)
{ return rsq >= P.maxsepsq && rsq >= (P.maxsep + s) * (P.maxsep + s); }

// FP32 decisions.  Each comparison a < b is made with a relative margin: inside the margin
// the entry is left to the FP64 code above, so every decision taken here equals the FP64
// one.  Margins: 1e-5 for plain comparisons (FP32 rounding of rsq, s and the constants is
// below 1e-6), 2e-4 where the fractional bin position enters (its FP32 error is below 1e-5).
__device__ __forceinline__ int lt3(float a, float b, float m)
{
    const float d = m * (fabsf(a) + fabsf(b));
    if (a < b - d) return 1;
    if (a > b + d) return 0;
    return -1;
}

// One (c1, c2) entry of a multipoleFinish pass in FP32.  Returns -1 (undecided: use FP64),
// 0 (dropped: too small, too large, or accepted outside [min_sep, max_sep)), 1 (accepted
// into bin k; r and logr returned) or 2 (not accepted: split flags, any = split1 and
// r + s > thresh1, r returned).
__device__ __forceinline__ int mp_decide32(const MPParams& P, float rsq, float s1, float s2,
                                           float thresh1, int& k, float& r, float& logr,
                                           bool& split1, bool& split2, bool& any)
{
    constexpr float M5 = 1e-5f, ML = 2e-4f;
    const float s = s1 + s2;
    // tooSmallDist: rsq < min_sep^2 && s < min_sep && rsq < (min_sep - s)^2.  min_sep - s
    // loses relative accuracy when s is close to min_sep: those go to FP64.
    const int below_min = lt3(rsq, P.f_minsepsq, M5);
    if (below_min < 0) return -1;
    if (below_min == 1) {
        const int c2 = lt3(s, P.f_minsep, M5);
        if (c2 < 0) return -1;
        if (c2 == 1) {
            const float d = P.f_minsep - s;
            if (d < 0.01f * P.f_minsep) return -1;
            const int c3 = lt3(rsq, d * d, ML);
            if (c3 < 0) return -1;
            if (c3 == 1) return 0;
        }
    }
    const int below_max = lt3(rsq, P.f_maxsepsq, M5);
    if (below_max < 0) return -1;
    if (below_max == 0) {                       // tooLargeDist
        const float ms = P.f_maxsep + s;
        const int c = lt3(rsq, ms * ms, M5);
        if (c < 0) return -1;
        if (c == 0) return 0;
    }
    // BinTypeHelper<Log>::singleBin
    bool sb;
    int ik = -1;
    float lr = 0.f;
    if (s == 0.f) {
        sb = true;
    } else {
        const float s2q = s * s;
        int c = lt3(P.f_asq * rsq, s2q, M5);
        if (c < 0) return -1;
        if (c == 1) {
            sb = false;
        } else {
            c = lt3(P.f_bsq * rsq, s2q, M5);
            if (c < 0) return -1;
            if (c == 0) {
                sb = true;
            } else {
                c = lt3(P.f_q25 * rsq, s2q, M5);
                if (c < 0) return -1;
                if (c == 1) {
                    sb = false;
                } else {
                    lr = 0.5f * logf(rsq);
                    const float kk = (lr - P.f_logminsep) / P.f_binsize;
                    ik = (int)kk;
                    const float frac = kk - (float)ik;
                    const float af = fabsf(frac);      // kk < 0 below min_sep: frac <= 0
                    if (af < ML || af > 1.f - ML) return -1;
                    const float f = fminf(frac, 1.f - frac);
                    const float t4 = f * P.f_binsize + P.f_b;
                    c = lt3(t4 * t4 * rsq, s2q, ML);
                    if (c < 0) return -1;
                    if (c == 1) {
                        sb = false;
                    } else {
                        const float t5 = frac * P.f_binsize + P.f_b - s2q / rsq;
                        c = lt3(t5 * t5 * rsq, s2q, ML);
                        if (c < 0) return -1;
                        sb = (c != 1);
                    }
                }
            }
        }
    }
    r = sqrtf(rsq);
    if (sb) {
        if (below_max == 0 || below_min == 1) return 0;   // isRSqInRange fails
        if (ik < 0) {
            lr = logf(r);
            const float kk = (lr - P.f_logminsep) / P.f_binsize;
            ik = (int)kk;
            const float frac = kk - (float)ik;
            if (frac < ML || frac > 1.f - ML) return -1;
        }
        k = ik < P.nbd ? ik : P.nbd - 1;
        logr = lr;
        return 1;
    }
    // CalcSplitSq (include/Split.h:82-101); s1, s2 are the cells' float sizes, so the size
    // comparisons are exact.
    const float bsq_eff = rsq * P.f_minba;
    if (s2 > s1) {
        split2 = true;
        if (s2 > 2.f * s1) split1 = false;
        else {
            const int c = lt3(0.3422f * bsq_eff, s1 * s1, M5);
            if (c < 0) return -1;
            split1 = (c == 1);
        }
    } else {
        split1 = true;
        if (s1 > 2.f * s2) split2 = false;
        else {
            const int c = lt3(0.3422f * bsq_eff, s2 * s2, M5);
            if (c < 0) return -1;
            split2 = (c == 1);
        }
    }
    any = false;
    if (split1) {
        const int c = lt3(thresh1, r + s, M5);
        if (c < 0) return -1;
        any = (c == 1);
    }
    return 2;
}

// calculate_direction(p1, p2) of include/ProjectHelper.h:272-345 (unnormalised).
__device__ __forceinline__ C2 direction(double x1, double y1, double z1, double x2, double y2,
                                        double z2)
{
    double dsq = (x1 - x2) * (x1 - x2) + (y1 - y2) * (y1 - y2) + (z1 - z2) * (z1 - z2);
    double cosA = (z1 - z2) + 0.5 * z2 * dsq;
    double sinA = y1 * x2 - x1 * y2;
    return {sinA, -cosA};
}

// ExpIPhi (ProjectHelper.h:264-266, 526-535, 688-697) and the spin-2 projection factor
// conj(r^2)/|r|^2 of ProjectWithSq, for the pair (c1, c2).
__device__ __forceinline__ void phases(const MPParams& P, int i, int j, double r, C2& z, C2& e)
{
    if (P.coords == FLAT) {
        double dx = P.x[j] - P.x[i], dy = P.y[j] - P.y[i];
        z = {dx / r, dy / r};
        double n = dx * dx + dy * dy;
        if (!(n > 0.)) n = 1.;
        e = {(dx * dx - dy * dy) / n, -(2. * dx * dy) / n};
        return;
    }
    double x1 = P.x[i], y1 = P.y[i], z1 = P.z[i], x2 = P.x[j], y2 = P.y[j], z2 = P.z[j];
    if (P.coords == THREED) { norm3(x1, y1, z1); norm3(x2, y2, z2); }
    C2 d = direction(x2, y2, z2, x1, y1, z1);
    double n = d.re * d.re + d.im * d.im;
    if (!(n > 0.)) n = 1.;
    double sn = sqrt(n);
    z = {d.re / sn, d.im / sn};
    C2 q = direction(x1, y1, z1, x2, y2, z2);
    double m = q.re * q.re + q.im * q.im;
    if (!(m > 0.)) m = 1.;
    e = {(q.re * q.re - q.im * q.im) / m, -(2. * q.re * q.im) / m};
}

// ---------------------------------------------------------------------------------------
// Block helpers.

__device__ __forceinline__ int block_excl_scan(int v, int* sh, int& total)
{
    // sh: MW ints.
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    int pre = 0;
    total = 0;
    for (int k = 0; k < MW; ++k) {
        if (k < wid) pre += sh[k];
        total += sh[k];
    }
    __syncthreads();
    return pre + x - v;
}

__device__ __forceinline__ void set_mp_err(int* err, int code) { atomicCAS(err, 0, code); }

// A consistency check that failed: record the site, the caller skips the item.
__device__ __forceinline__ void mp_check_fail(int* err, int site)
{
    atomicCAS(err, 0, MP_ERR_CHECK);
    atomicCAS(err + 1, 0, site);
}

__device__ __forceinline__ bool mp_valid_cell(const MPParams& P, int c)
{ return c >= 0 && c < P.ncells && P.n[c] > 0; }

// ---------------------------------------------------------------------------------------
// Phase 1: multipoleSplit1 + splitC2Cells, one block per vertex-1 top-level cell; its pair
// list starts as all top cells of the pair field (the same field for an auto-correlation,
// src/Corr3.cpp:1124-1175; field 2 for cross12, 1177-1237).

struct P1Entry { int c1, off, len, pad; };

__global__ void __launch_bounds__(MB) k_mp_split1(MPParams P)
{
    __shared__ P1Entry stk[MSTACK];
    __shared__ int sp, top_rel, scan_sh[MW], have_sh;
    __shared__ P1Entry cur;
    const int b = blockIdx.x;
    int* arena = P.arena1 + (size_t)b * P.arena1_cap;
    const int tid = threadIdx.x;
    for (int j = tid; j < P.ntop2; j += MB) arena[j] = P.tops2[j];
    if (tid == 0) {
        sp = 0;
        top_rel = P.ntop2;
        stk[sp++] = {P.tops[b], 0, P.ntop2, 0};
    }
    __syncthreads();
    int guard = 0;
    while (true) {
        // Thread 0 pops; everyone learns the outcome from a flag written before the barrier
        // (reading sp directly would race with the pop).
        __syncthreads();
        if (tid == 0) {
            have_sh = sp > 0;
            if (have_sh) cur = stk[--sp];
        }
        __syncthreads();
        if (!have_sh) break;
        if (++guard > (1 << 24)) {
            if (tid == 0) set_mp_err(P.err, MP_ERR_STACK);
            break;
        }
        const int c1 = cur.c1;
        const double s1 = P.size[c1];
        const int base = top_rel;
        int written = 0;
        for (int j0 = 0; j0 < cur.len; j0 += MB) {
            const int j = j0 + tid;
            int cnt = 0, ca = -1, cb = -1;
            const int c2 = j < cur.len ? __ldcg(arena + cur.off + j) : 0;
            if (j < cur.len && !mp_valid_cell(P, c2)) mp_check_fail(P.err, 1);
            else if (j < cur.len) {
                const double s2 = P.size[c2];
                const double rsq = mp_dist_sq(P, c1, c2);
                const double s = s1 + s2;
                if (!mp_too_small(P, rsq, s) && !mp_too_large(P, rsq, s)) {
                    int k = -1;
                    double r = 0., lr = 0.;
                    bool split = !mp_single_bin(P, rsq, s, k, r, lr);
                    if (split && s2 > s1) { ca = P.left[c2]; cb = P.right[c2]; cnt = 2; }
                    else { ca = c2; cnt = 1; }
                }
            }
            int total;
            int pos = block_excl_scan(cnt, scan_sh, total);
            if (base + written + total > P.arena1_cap) {
                if (tid == 0) set_mp_err(P.err, MP_ERR_ARENA);
            } else {
                if (cnt >= 1) arena[base + written + pos] = ca;
                if (cnt == 2) arena[base + written + pos + 1] = cb;
            }
            written += total;
        }
        __syncthreads();
        if (base + written > P.arena1_cap) break;   // overflow flagged: lists incomplete
        if (tid == 0) {
            top_rel = base + written;
            if ((double)s1 * (double)s1 > P.maxbsq_eff && P.left[c1] >= 0) {
                if (sp + 2 > MSTACK) set_mp_err(P.err, MP_ERR_STACK);
                else {
                    stk[sp++] = {P.right[c1], base, written, 0};
                    stk[sp++] = {P.left[c1], base, written, 0};
                }
            } else {
                unsigned long long jn = atomicAdd(P.njobs, 1ull);
                if ((long long)jn < P.jobs_cap) P.jobs[jn] = make_int4(c1, b, base, written);
                else set_mp_err(P.err, MP_ERR_JOBS);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Phase 2: multipoleFinish per job.

// maxr / maxr3: the previous pass's largest remaining r + s over the vertex-2 (or only)
// list and the vertex-3 list (multipoleFinish keeps them apart, src/Corr3.cpp:1616-1679).
struct P2Entry { int c1, len, slot, mink; long long goff; double maxr, maxr3; long long mark; };

// Scratch slot layout (doubles): W_n [n = 0 .. M][bin] complex, G_n [n + M + 1 = 0 .. 2M+2]
// [bin] complex, gg0/gg1/gg2 [bin] complex, then npairs, sumw, sumwr, sumwlogr, sumww,
// sumwwr, sumwwlogr [bin].  The [n][bin] order is the vertex record's order.
__device__ __forceinline__ size_t sW(int nb, int n, int k) { return 2 * ((size_t)n * nb + k); }
__device__ __forceinline__ size_t sG(int nb, int M, int n, int k)
{ return 2 * ((size_t)(n + M + 1) * nb + k); }
__device__ __forceinline__ double* slot_ptr(const MPParams& P, int blk, int s)
{ return P.slots + ((size_t)blk * P.nslots + s) * P.slot_doubles; }

// Accepted-pair record (MP_REC floats): z (2), wg = g2 * e (2), w2, n2 (int), k (int), pad,
// then the 14 scalar terms of calculateGn: w2, w2 r, w2 logr, sum w^2, (sum w^2) r,
// (sum w^2) logr, sumwwgg0 (2), sumwwgg1 (2), sumwwgg2 (2), wg (2).
static constexpr int REC_K = 6;

// A warp's staged batch of 32 records: powers of z (16 records at a time), (wg, w2, bin), scalar
// terms (14, n2, w2).
struct AccBatch {
    float2 pw[16][33];
    float4 hk[32];
    float sc[32][17];
};
static_assert(sizeof(AccBatch) % 16 == 0, "");

// Bin-ordered G_n / W_n accumulation of the records [0, nrec) of this block into slot S.
// The records are ranked by bin, then warp w takes the w-th contiguous share of the ranked
// records, 32 at a time: two lanes write a record's powers z .. z^16 and z^17 .. z^32 (z^33 .. in
// a second round, H = 2) to shared memory, one complex multiplication each, and the record's
// other terms, 16 records at a time; then lane = n walks the records of each bin's run with six FP32 multiply-adds each (the sums of
// Re wg z^n and Im wg z^n, which make both G_n and G_-n, and w z^n), lanes 0..15 adding
// the scalar terms as well.  The FP32 sums (F over a batch, F2 over the share: at most 1024
// records, so 32 batches) go to the slot in FP64 when the bin changes (atomics: two warps can share a bin).
// A record costs the warp 22 instructions; raising every lane to its own power by squaring
// took 75.
template <int H>
__device__ __forceinline__ void mp_accumulate(const MPParams& P, const float* rec, int* perm, int nrec,
                              double* S, int* bh, AccBatch* batches)
{
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nb = P.nbins, M = P.maxn, gst = 2 * M + 3;
    // Ranking by bin: bh holds the per-bin counts on entry.
    if (wid == 0) {
        int total = 0;
        for (int k0 = 0; k0 < nb; k0 += 32) {
            const int c = k0 + lane < nb ? bh[k0 + lane] : 0;
            int x = c;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (k0 + lane < nb) bh[k0 + lane] = total + x - c;
            total += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0 && total != nrec) mp_check_fail(P.err, 8);   // counts and records disagree
    }
    __syncthreads();
    for (int c0 = 32 * wid; c0 < nrec; c0 += MB) {
        const int a = c0 + lane;
        const int k = a < nrec ? __float_as_int(__ldcg(rec + (size_t)a * MP_REC + REC_K)) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, k);
        const int leader = __ffs(peers) - 1;
        int pos = 0;
        if (lane == leader && k >= 0 && k < nb) pos = atomicAdd(&bh[k], __popc(peers));
        pos = __shfl_sync(0xffffffffu, pos, leader) + __popc(peers & ((1u << lane) - 1u));
        if (k >= 0 && pos < nrec) perm[pos] = a;
    }
    __syncthreads();
    for (int k = tid; k < nb; k += MB) bh[k] = 0;   // counts of the next batch
    double* W = S;
    double* G = S + 2 * (size_t)nb * (M + 1);
    const int per = (nrec + MW - 1) / MW;
    const int p0 = wid * per, p1 = min(nrec, p0 + per);
    AccBatch& B = batches[wid];
    // This lane's scalar sum in the slot: place for bin 0 and step per bin.
    const int oG = 2 * nb * (M + 1), oGG = oG + 2 * nb * gst, oSC = oGG + 6 * nb;
    int sc0 = 0, scs = 1;
    if (lane < 6) sc0 = oSC + (lane + 1) * nb;
    else if (lane < 12) { sc0 = oGG + ((lane - 6) >> 1) * 2 * nb + (lane & 1); scs = 2; }
    else if (lane < 14) { sc0 = oG + (int)sG(nb, M, 0, 0) + lane - 12; scs = 2; }
    else if (lane == 14) sc0 = oSC;
    else { sc0 = (int)sW(nb, 0, 0); scs = 2; }
    float F[H][6], F2[H][6], fs = 0.f, fs2 = 0.f;
    unsigned cn = 0;
    int curk[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
        curk[h] = -1;
#pragma unroll
        for (int q = 0; q < 6; ++q) { F[h][q] = 0.f; F2[h][q] = 0.f; }
    }
    auto flush = [&](int h, int k) {
        const int n = lane + 1 + 32 * h;
        float* f = F[h];
        float* f2 = F2[h];
#pragma unroll
        for (int q = 0; q < 6; ++q) { f2[q] += f[q]; f[q] = 0.f; }
        if (n <= M) {
            double* wp = W + sW(nb, n, k);
            atomicAdd(wp, (double)f2[0]);
            atomicAdd(wp + 1, (double)f2[1]);
        }
        if (n <= M + 1) {
            double* gp = G + sG(nb, M, n, k);
            double* gm = G + sG(nb, M, -n, k);
            atomicAdd(gp, (double)(f2[2] - f2[5]));
            atomicAdd(gp + 1, (double)(f2[3] + f2[4]));
            atomicAdd(gm, (double)(f2[2] + f2[5]));
            atomicAdd(gm + 1, (double)(f2[4] - f2[3]));
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) f2[q] = 0.f;
        if (h == 0) {
            if (lane < 16) atomicAdd(S + sc0 + (size_t)scs * k, lane == 14 ? (double)cn : (double)(fs2 + fs));
            fs = fs2 = 0.f;
            cn = 0;
        }
    };
    for (int base = p0; base < p1; base += 32) {
        const int nv = min(32, p1 - base);
        const bool in = lane < nv;
        const int pi = in ? __ldcg(perm + base + lane) : 0;
        const bool bad = pi < 0 || pi >= nrec;          // every rank is filled exactly once
        if (bad) mp_check_fail(P.err, 4);
        const float4* r4 = reinterpret_cast<const float4*>(rec + (size_t)(bad ? 0 : pi) * MP_REC);
        const float4 h0 = __ldcg(r4), h1 = __ldcg(r4 + 1), q0 = __ldcg(r4 + 2), q1 = __ldcg(r4 + 3);
        const float4 q2 = __ldcg(r4 + 4), q3 = __ldcg(r4 + 5);
        int k = __float_as_int(h1.z);
        if (k < 0 || k >= nb) { mp_check_fail(P.err, 5); k = 0; }
        const int kp = __shfl_up_sync(0xffffffffu, k, 1);
        const unsigned starts = __ballot_sync(0xffffffffu, in && lane > 0 && k != kp);
        __syncwarp();                                   // the batch before has been read
        B.hk[lane] = make_float4(h0.z, h0.w, h1.x, __int_as_float(k));
        {
            const float sv[16] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w,
                                  q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, h1.y, h1.x};
#pragma unroll
            for (int q = 0; q < 16; ++q) B.sc[lane][q] = sv[q];
        }
        // Records 0..15, then 16..31; two lanes to a record, for the lower and the upper 16 powers.
        for (int r0 = 0; r0 < nv; r0 += 16) {
            const int rec16 = lane & 15, up = lane >> 4, jend = min(nv, r0 + 16);
            const float zr = __shfl_sync(0xffffffffu, h0.x, r0 + rec16);
            const float zi = __shfl_sync(0xffffffffu, h0.y, r0 + rec16);
            float sr = zr, si = zi;                     // z^16
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float u = sr * sr - si * si;
                si = 2.f * sr * si;
                sr = u;
            }
            float pr = up ? sr : 1.f, pi2 = up ? si : 0.f;
#pragma unroll
            for (int h = 0; h < H; ++h) {
                if (h == 1) {                           // from z^16 on: another z^16
                    const float t = pr * sr - pi2 * si;
                    pi2 = pr * si + pi2 * sr;
                    pr = t;
                }
                const int nc = min(16, M + 1 - 32 * h - 16 * up);
                if (r0 + h > 0) __syncwarp();
#pragma unroll 4
                for (int n = 0; n < nc; ++n) {
                    const float t = pr * zr - pi2 * zi;
                    pi2 = pr * zi + pi2 * zr;
                    pr = t;
                    B.pw[rec16][16 * up + n] = make_float2(pr, pi2);
                }
                __syncwarp();
                for (int js = r0; js < jend;) {
                    const unsigned later = js < 31 ? starts & ~((2u << js) - 1u) : 0u;
                    const int je = min(later ? __ffs(later) - 1 : nv, jend);
                    const int kj = __float_as_int(B.hk[js].w);
                    if (kj != curk[h]) {
                        if (curk[h] >= 0) flush(h, curk[h]);
                        curk[h] = kj;
                    }
#pragma unroll 4
                    for (int j = js; j < je; ++j) {
                        const float2 z = B.pw[j & 15][lane];
                        const float4 hk = B.hk[j];
                        F[h][0] = fmaf(hk.z, z.x, F[h][0]);
                        F[h][1] = fmaf(hk.z, z.y, F[h][1]);
                        F[h][2] = fmaf(hk.x, z.x, F[h][2]);     // Re wg Re z^n
                        F[h][3] = fmaf(hk.x, z.y, F[h][3]);     // Re wg Im z^n
                        F[h][4] = fmaf(hk.y, z.x, F[h][4]);     // Im wg Re z^n
                        F[h][5] = fmaf(hk.y, z.y, F[h][5]);     // Im wg Im z^n
                        if (h == 0) {
                            const float v = B.sc[j][lane & 15];
                            fs += v;
                            cn += __float_as_uint(v);           // (lane 14: the point count)
                        }
                    }
                    js = je;
                }
            }
        }
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int q = 0; q < 6; ++q) { F2[h][q] += F[h][q]; F[h][q] = 0.f; }
        fs2 += fs;
        fs = 0.f;
    }
#pragma unroll
    for (int h = 0; h < H; ++h)
        if (curk[h] >= 0) flush(h, curk[h]);
    __syncthreads();
}

// The n = 0 scalar outputs of calculateZeta for rows k2 in [ks, mk): ntri, meand2/3,
// meanlogd2/3 (FP64 atomics into the outputs).
__device__ void zeta_scalars(const MPParams& P, int c1, const double* S, int ks, int mk,
                             double* out)
{
    const int nb = P.nbins, M = P.maxn, nn = 2 * M + 1;
    const int gst = 2 * M + 3;
    const size_t Z = (size_t)nb * nb * nn;
    const double* SC = S + 2 * (size_t)nb * (M + 1) + 2 * (size_t)nb * gst + 6 * (size_t)nb;
    // The slot was just updated by atomics: read it from L2.
    auto npairs = [&](int k) { return __ldcg(SC + k); };
    auto sumw = [&](int k) { return __ldcg(SC + nb + k); };
    auto sumwr = [&](int k) { return __ldcg(SC + 2 * nb + k); };
    auto sumwlogr = [&](int k) { return __ldcg(SC + 3 * nb + k); };
    auto sumwwr = [&](int k) { return __ldcg(SC + 5 * nb + k); };
    auto sumwwlogr = [&](int k) { return __ldcg(SC + 6 * nb + k); };
    const double w1 = P.w[c1];
    const double n1 = P.n[c1];
    const int rows = mk - ks;
    for (int t = threadIdx.x; t < rows * nb; t += MB) {
        const int k2 = ks + t / nb, k3 = t % nb;
        if (k3 < k2) continue;
        const int i23 = (k2 * nb + k3) * nn + M;
        if (k3 == k2) {
            atomicAdd(&out[14 * Z + i23], n1 * npairs(k2) * (npairs(k2) - 1));
            double md = w1 * (sumw(k2) * sumwr(k2) - sumwwr(k2));
            double ml = w1 * (sumw(k2) * sumwlogr(k2) - sumwwlogr(k2));
            atomicAdd(&out[8 * Z + i23], md); atomicAdd(&out[9 * Z + i23], ml);
            atomicAdd(&out[10 * Z + i23], md); atomicAdd(&out[11 * Z + i23], ml);
        } else {
            const int i32 = (k3 * nb + k2) * nn + M;
            double nnn = n1 * npairs(k2) * npairs(k3);
            atomicAdd(&out[14 * Z + i23], nnn); atomicAdd(&out[14 * Z + i32], nnn);
            double ww12 = w1 * sumw(k2), ww13 = w1 * sumw(k3);
            atomicAdd(&out[8 * Z + i23], ww13 * sumwr(k2));  atomicAdd(&out[10 * Z + i32], ww13 * sumwr(k2));
            atomicAdd(&out[9 * Z + i23], ww13 * sumwlogr(k2)); atomicAdd(&out[11 * Z + i32], ww13 * sumwlogr(k2));
            atomicAdd(&out[10 * Z + i23], ww12 * sumwr(k3)); atomicAdd(&out[8 * Z + i32], ww12 * sumwr(k3));
            atomicAdd(&out[11 * Z + i23], ww12 * sumwlogr(k3)); atomicAdd(&out[9 * Z + i32], ww12 * sumwlogr(k3));
        }
    }
}

// The self-pair corrections of the diagonal entries k2 == k3 (the same for every n), rows
// [ks, mk): gam0 -= wg1 sumwwgg0, gam1 -= conj(wg1) sumwwgg1, gam2, gam3 -= wg1 sumwwgg2,
// weight -= w1 sumww.  Stored positive in the block's diag array and subtracted at the end.
__device__ void zeta_diag(const MPParams& P, int c1, const double* S, int ks, int mk,
                          double* diag)
{
    const int nb = P.nbins, M = P.maxn, gst = 2 * M + 3;
    const double* GG = S + 2 * (size_t)nb * (M + 1) + 2 * (size_t)nb * gst;
    const double* sumww = GG + 6 * (size_t)nb + 4 * (size_t)nb;
    const double w1 = P.w[c1];
    const C2 wg1 = {(double)P.d1[c1], (double)P.d2[c1]};
    for (int a = ks + threadIdx.x; a < mk; a += MB) {
        const C2 t0 = cmul(wg1, {__ldcg(GG + 2 * a), __ldcg(GG + 2 * a + 1)});
        const C2 t1 = cmul(conj2(wg1), {__ldcg(GG + 2 * nb + 2 * a), __ldcg(GG + 2 * nb + 2 * a + 1)});
        const C2 t2 = cmul(wg1, {__ldcg(GG + 4 * nb + 2 * a), __ldcg(GG + 4 * nb + 2 * a + 1)});
        // (this block's own sums; atomics only so that no thread waits for a load)
        const double v[9] = {t0.re, t0.im, t1.re, t1.im, t2.re, t2.im, t2.re, t2.im, w1 * __ldcg(sumww + a)};
#pragma unroll
        for (int q = 0; q < 9; ++q) atomicAdd(diag + q * nb + a, v[q]);
    }
}

// The product terms of calculateZeta for the entries (a, b, n) with min(a, b) in [ks, mk),
// in FP64 directly into the outputs (atomics): the path for a vertex record that does not fit
// the record buffer.
__device__ void zeta_products(const MPParams& P, int c1, const double* S, int ks, int mk,
                              double* out, double* shG, double* shW)
{
    const int nb = P.nbins, M = P.maxn, nn = 2 * M + 1;
    const int gst = 2 * M + 3;
    const size_t Z = (size_t)nb * nb * nn;
    const double* W = S;
    const double* G = S + 2 * (size_t)nb * (M + 1);
    for (int q = threadIdx.x; q < 2 * nb * gst; q += MB) shG[q] = __ldcg(G + q);
    for (int q = threadIdx.x; q < 2 * nb * (M + 1); q += MB) shW[q] = __ldcg(W + q);
    __syncthreads();
    const double w1 = P.w[c1];
    const C2 wg1 = {(double)P.d1[c1], (double)P.d2[c1]};
    const C2 wg1c = conj2(wg1);
    auto Gv = [&](int k, int n) -> C2 {
        const double* p = shG + sG(nb, M, n, k);
        return {p[0], p[1]};
    };
    auto Wv = [&](int k, int n) -> C2 {
        const double* p = shW + sW(nb, n >= 0 ? n : -n, k);
        return n >= 0 ? C2{p[0], p[1]} : C2{p[0], -p[1]};
    };
    const int na = mk - ks;
    const long long cnt = (long long)na * nb * 2 * nn;   // pairs (a in rows, b >= a) and mirror
    for (long long t = threadIdx.x; t < cnt; t += MB) {
        const int n = (int)(t % nn) - M;
        long long rest = t / nn;
        const int mirror = (int)(rest % 2);
        rest /= 2;
        const int bb = (int)(rest % nb);
        const int aa = ks + (int)(rest / nb);
        if (bb < aa) continue;                     // (aa, bb) with bb >= aa; the mirror swaps
        if (bb == aa && mirror) continue;
        const int a = mirror ? bb : aa, b = mirror ? aa : bb;
        const size_t i = (size_t)(a * nb + b) * nn + M + n;
        // weight (Porth et al. eq. 27)
        if (a == b) {
            C2 wv = Wv(a, n);
            atomicAdd(&out[12 * Z + i], w1 * (wv.re * wv.re + wv.im * wv.im));
        } else {
            C2 p = cmul(Wv(a, n), conj2(Wv(b, n)));
            atomicAdd(&out[12 * Z + i], w1 * p.re);
            atomicAdd(&out[13 * Z + i], w1 * p.im);
        }
        // gam0..3 (eqs. 21, 23-25)
        C2 g0 = cmul(cmul(wg1, Gv(a, n - 1)), Gv(b, -n - 1));
        C2 g1 = cmul(cmul(wg1c, Gv(a, n + 1)), Gv(b, -n + 1));
        C2 g2 = cmul(cmul(wg1, Gv(a, n - 1)), conj2(Gv(b, n + 1)));
        C2 g3 = cmul(cmul(wg1, conj2(Gv(a, -n + 1))), Gv(b, -n - 1));
        atomicAdd(&out[0 * Z + i], g0.re); atomicAdd(&out[1 * Z + i], g0.im);
        atomicAdd(&out[2 * Z + i], g1.re); atomicAdd(&out[3 * Z + i], g1.im);
        atomicAdd(&out[4 * Z + i], g2.re); atomicAdd(&out[5 * Z + i], g2.im);
        atomicAdd(&out[6 * Z + i], g3.re); atomicAdd(&out[7 * Z + i], g3.im);
    }
    __syncthreads();
}

// The in-place path of a three-field cross (Corr3::calculateZeta with mp2, mp3,
// src/Corr3.cpp:1976-2087): every entry (a, b) of the scratch's 2 nbd x 2 nbd bins whose
// row and column belong to different vertices and whose min(a mod nbd, b mod nbd) is in
// [ks, mk), with the auto-correlation's off-diagonal formulas; the caller keeps the
// vertex-3 x vertex-2 block (and, for ordered = 1, adds the other).
__device__ void zeta_inplace3(const MPParams& P, int c1, const double* S, int ks, int mk,
                              double* out, double* shG, double* shW)
{
    const int nb = P.nbins, nbd = P.nbd, M = P.maxn, nn = 2 * M + 1;
    const int gst = 2 * M + 3;
    const size_t Z = (size_t)nb * nb * nn;
    const double* W = S;
    const double* G = S + 2 * (size_t)nb * (M + 1);
    const double* SC = G + 2 * (size_t)nb * gst + 6 * (size_t)nb;
    for (int q = threadIdx.x; q < 2 * nb * gst; q += MB) shG[q] = __ldcg(G + q);
    for (int q = threadIdx.x; q < 2 * nb * (M + 1); q += MB) shW[q] = __ldcg(W + q);
    __syncthreads();
    const double w1 = P.w[c1];
    const double n1 = P.n[c1];
    const C2 wg1 = {(double)P.d1[c1], (double)P.d2[c1]};
    const C2 wg1c = conj2(wg1);
    const int sh = P.vreal ? 0 : 1;
    auto Gv = [&](int k, int n) -> C2 {
        const double* p = shG + sG(nb, M, n, k);
        return {p[0], p[1]};
    };
    auto Wv = [&](int k, int n) -> C2 {
        const double* p = shW + sW(nb, n >= 0 ? n : -n, k);
        return n >= 0 ? C2{p[0], p[1]} : C2{p[0], -p[1]};
    };
    const long long cnt = (long long)nb * nb * nn;
    for (long long t = threadIdx.x; t < cnt; t += MB) {
        const int n = (int)(t % nn) - M;
        const int b = (int)((t / nn) % nb), a = (int)(t / nn / nb);
        if ((a >= nbd) == (b >= nbd)) continue;
        const int m = min(a % nbd, b % nbd);
        if (m < ks || m >= mk) continue;
        const size_t i = (size_t)(a * nb + b) * nn + M + n;
        const C2 p = cmul(Wv(a, n), conj2(Wv(b, n)));
        atomicAdd(&out[12 * Z + i], w1 * p.re);
        atomicAdd(&out[13 * Z + i], w1 * p.im);
        const C2 g0 = cmul(cmul(wg1, Gv(a, n - sh)), Gv(b, -n - sh));
        const C2 g1 = cmul(cmul(wg1c, Gv(a, n + sh)), Gv(b, -n + sh));
        const C2 g2 = cmul(cmul(wg1, Gv(a, n - sh)), conj2(Gv(b, n + sh)));
        const C2 g3 = cmul(cmul(wg1, conj2(Gv(a, -n + sh))), Gv(b, -n - sh));
        atomicAdd(&out[0 * Z + i], g0.re); atomicAdd(&out[1 * Z + i], g0.im);
        atomicAdd(&out[2 * Z + i], g1.re); atomicAdd(&out[3 * Z + i], g1.im);
        atomicAdd(&out[4 * Z + i], g2.re); atomicAdd(&out[5 * Z + i], g2.im);
        atomicAdd(&out[6 * Z + i], g3.re); atomicAdd(&out[7 * Z + i], g3.im);
        if (n == 0 && !P.quick) {
            const size_t i0 = (size_t)(a * nb + b) * nn + M;
            const double npa = __ldcg(SC + a), npb = __ldcg(SC + b);
            const double swa = __ldcg(SC + nb + a), swb = __ldcg(SC + nb + b);
            const double sra = __ldcg(SC + 2 * nb + a), srb = __ldcg(SC + 2 * nb + b);
            const double sla = __ldcg(SC + 3 * nb + a), slb = __ldcg(SC + 3 * nb + b);
            // meanlogd3 of the vertex-3 x vertex-2 block for ordered = 1 as the reference
            // writes it: mp3.sumw at the column's bin.
            const double swl = (P.typo32 && a >= nbd) ? __ldcg(SC + nb + (b % nbd) + nbd) : swa;
            atomicAdd(&out[14 * Z + i0], n1 * npa * npb);
            atomicAdd(&out[8 * Z + i0], w1 * swb * sra);
            atomicAdd(&out[9 * Z + i0], w1 * swb * sla);
            atomicAdd(&out[10 * Z + i0], w1 * swa * srb);
            atomicAdd(&out[11 * Z + i0], w1 * swl * slb);
        }
    }
    __syncthreads();
}

// calculateZeta for vertex c1, rows [ks, mk): the diagonal self-pair corrections now, the
// rest as one vertex record for the batched contraction kernels (k_mp_zeta, k_mp_zscal).
// Record (floats): header (c1, ks, mk, w1, Re/Im wg1, n1, pad), then npairs (int), sumw, sumwr,
// sumwlogr, sumwwr, sumwwlogr [bin], then G_n [n = -(M+1) .. M+1][bin] and W_n [n = 0 ..
// M][bin] complex, of the bins from ks on (min(a, b) >= ks; all bins of a three-field cross).
// A record that does not fit the buffer is contracted in place.
__device__ void zeta_emit(const MPParams& P, int c1, const double* S, int ks, int mk,
                          double* out, double* diag, double* shG, double* shW,
                          unsigned long long* zidx_sh, int* emits_sh)
{
    const int nb = P.nbins, M = P.maxn, gst = 2 * M + 3;
    // (number, 16-byte offset), in one counter
    const int c0 = P.three ? 0 : ks, nc = nb - c0, total = (gst + M + 1) * nc;
    const long long units = (8 + 6 * nb + 2 * total + 3) / 4;
    if (threadIdx.x == MB - 1) {
        *zidx_sh = atomicAdd(P.zcount, ZC_ONE + (unsigned long long)units);
        ++*emits_sh;
    }
    // G's rows, then W's, eight columns per thread in flight.
    const double2* W = reinterpret_cast<const double2*>(S);
    const double2* G = W + (size_t)nb * (M + 1);
    const int dr = MB / nc, dc = MB - dr * nc;
    int row = threadIdx.x / nc, col = threadIdx.x - row * nc;
    double2 v[8];
    auto load8 = [&](int q0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (q0 + u * MB < total)
                v[u] = __ldcg((row < gst ? G + (size_t)row * nb : W + (size_t)(row - gst) * nb) + c0 + col);
            row += dr;
            col += dc;
            if (col >= nc) { col -= nc; ++row; }
        }
    };
    // (a three-field cross has no self-pair corrections: getMP2 / getMP3 without ww)
    if (!P.three) zeta_diag(P, c1, S, ks, mk, diag);
    __syncthreads();
    const long long zi = (long long)(*zidx_sh / ZC_ONE), off = (long long)(*zidx_sh % ZC_ONE);
    const bool fits = zi < P.zmax && off + units <= P.zcap;
    if (threadIdx.x == 0 && zi < P.zmax) P.zoff[zi] = fits ? (unsigned)off : ZOFF_NONE;
    if (fits) {
        float* R = P.zrec + 4 * (size_t)off;
        if (threadIdx.x == 0) {
            R[0] = __int_as_float(c1); R[1] = __int_as_float(ks); R[2] = __int_as_float(mk);
            R[3] = P.w[c1]; R[4] = P.d1[c1]; R[5] = P.d2[c1];
            R[6] = __int_as_float(P.n[c1]); R[7] = 0.f;
        }
        float2* RG = reinterpret_cast<float2*>(R + 8 + 6 * nb);
        for (int q0 = threadIdx.x; q0 < total; q0 += 8 * MB) {
            load8(q0);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (q0 + u * MB < total) RG[q0 + u * MB] = make_float2((float)v[u].x, (float)v[u].y);
        }
        const double* SC = S + 2 * (size_t)nb * (M + 1) + 2 * (size_t)nb * gst + 6 * (size_t)nb;
        float* RS = R + 8;
        for (int q = threadIdx.x; q < nb; q += MB) {
            RS[q] = __int_as_float((int)__ldcg(SC + q));                // npairs
            RS[nb + q] = (float)__ldcg(SC + nb + q);                    // sumw
            RS[2 * nb + q] = (float)__ldcg(SC + 2 * nb + q);            // sumwr
            RS[3 * nb + q] = (float)__ldcg(SC + 3 * nb + q);            // sumwlogr
            RS[4 * nb + q] = (float)__ldcg(SC + 5 * nb + q);            // sumwwr
            RS[5 * nb + q] = (float)__ldcg(SC + 6 * nb + q);            // sumwwlogr
        }
    } else if (P.three) {
        zeta_inplace3(P, c1, S, ks, mk, out, shG, shW);
    } else {
        if (!P.quick) zeta_scalars(P, c1, S, ks, mk, out);
        zeta_products(P, c1, S, ks, mk, out, shG, shW);
    }
    __syncthreads();
}

// No job is started once the buffer holds zstop units or zmaxstop records.
__device__ __forceinline__ bool zbuffer_full(const MPParams& P)
{
    const unsigned long long c = *(volatile unsigned long long*)P.zcount;
    return (long long)(c % ZC_ONE) >= P.zstop || (long long)(c / ZC_ONE) >= P.zmaxstop;
}

// Phase 2.  GGG of 500,000 points (20 bins, max_n 30) walks 1.87e6 lists of 908 cells on average,
// accepts 0.8e9 pairs and emits 1.57e6 vertex records: 373 ms before, 188 ms now (225 with 4 blocks
// an SM and 32 records' powers staged: 90 of it the lists' decisions, 85 the accumulation and 50
// the records).  What counts, as one SM has 20 warps here and every list is a chain of
// dependent loads and barriers:
//   * FP64: an instruction takes 16 cycles of the SM.  The largest r + s, the bin of its
//     logarithm and the block's maximum took a third of the time on all warps; now only the
//     threads that can hold the maximum leave FP32.
//   * one barrier per 128 list entries (places by ballots), none for the running counts;
//   * G_n, W_n rows copied and converted eight loads at a time, and only the record's columns;
//   * one buffer for all records: a wave's end costs the blocks' last jobs, 10 ms.
//   * shared memory and registers for 5 blocks of 128 threads (4: 232 ms for the call against 221);
//   * one array of outputs for what is contracted in place, not one per block to clear and sum.
// Taken back: the next entries loaded ahead (spills: 287 ms for the call against 254),
// mp_accumulate out of line (295), blocks of 256 threads (267 with two, 303 with three).
//
// THREE: a three-field cross (two pair lists); compiled apart so that the auto and cross12
// paths carry none of its registers.
template <bool THREE, int H>
__global__ void __launch_bounds__(MB, MBLK) k_mp_finish(const __grid_constant__ MPParams P)
{
    extern __shared__ __align__(16) double mp_sh[];
    __shared__ P2Entry stk[MSTACK];
    __shared__ int sp, free_cnt, free_list[64];
    __shared__ int2 scan_sh[2][MW];
    __shared__ P2Entry cur;
    __shared__ unsigned long long job_sh, zidx_sh, max_sh[2];
    __shared__ int alloc_ok, have_sh, job_emits;
    __shared__ unsigned best_sh[2][MW];     // warps' largest r + s (float bits); any split: bit 31
    __shared__ long long arena_top;
    __shared__ int bh[MP_MAXNB];
    AccBatch* batches = reinterpret_cast<AccBatch*>(mp_sh);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int blk = blockIdx.x;
    const int nb = P.nbins, M = P.maxn;
    const int gst = 2 * M + 3;
    double* shG = mp_sh;
    double* shW = mp_sh + 2 * (size_t)nb * gst;
    int* arena = P.arena2 + (size_t)blk * P.arena2_cap;
    float* acc = P.acc + (size_t)blk * P.acc_cap * MP_REC;
    int* perm = P.perm + (size_t)blk * P.acc_cap;
    double* out = P.out;
    double* diag = P.diag + (size_t)blk * 9 * nb;
    const int* arena1 = P.arena1;
    for (int k = tid; k < MP_MAXNB; k += MB) bh[k] = 0;

    while (true) {
        if (tid == 0) {
            // After an error the results are discarded and the call is retried: stop early.
            // With the vertex-record buffer nearly full, stop taking jobs until it is drained.
            if (*(volatile int*)P.err ||
                zbuffer_full(P))
                job_sh = (unsigned long long)P.njobs_val;
            else
                job_sh = atomicAdd(P.job_next, 1ull);
        }
        __syncthreads();
        const unsigned long long job = job_sh;
        if ((long long)job >= P.njobs_val) break;
        const int4 J = P.jobs[job];
        if (!mp_valid_cell(P, J.x) || J.y < 0 || J.y >= P.ntop || J.z < 0 || J.w < 0 ||
            (long long)J.z + J.w > P.arena1_cap) {
            if (tid == 0) mp_check_fail(P.err, 3);
            break;
        }
        if (tid == 0) {
            free_cnt = P.nslots;
            for (int s = 0; s < P.nslots; ++s) free_list[s] = P.nslots - 1 - s;
            arena_top = 0;
            sp = 0;
            job_emits = 0;
            int s0 = free_list[--free_cnt];
            P2Entry e;
            e.c1 = J.x; e.len = J.w; e.slot = s0; e.mink = P.nbd;
            e.goff = (long long)J.y * P.arena1_cap + J.z; e.maxr = 0.; e.maxr3 = 0.;
            e.mark = 0;
            stk[sp++] = e;
        }
        __syncthreads();
        int guard = 0, stall = 0, stall_c1 = -1;
        {
            double* S0 = slot_ptr(P, blk, stk[0].slot);
            for (int q = tid; q < P.slot_doubles; q += MB) S0[q] = 0.;
        }
        __syncthreads();
        while (true) {
            // Thread 0 pops (see k_mp_split1 for why the outcome goes through a flag).
            __syncthreads();
            if (tid == 0) {
                have_sh = sp > 0;
                if (have_sh) {
                    cur = stk[--sp];
                    arena_top = cur.mark;   // the finished left subtree's lists are dead
                }
            }
            __syncthreads();
            if (!have_sh) break;
            // multipoleFinish loop on cur (c1 changes to its left child, the list to the new
            // list, the slot stays).
            while (true) {
                if (++guard > (1 << 24)) {   // last-resort bound; the recursion is finite
                    if (tid == 0) mp_check_fail(P.err, 6);
                    break;
                }
                // Passes at one c1 refine its c2 list; their number is bounded by the depth
                // of the c2 trees.
                if (cur.c1 != stall_c1) { stall_c1 = cur.c1; stall = 0; }
                if (++stall > 4096) {
                    if (tid == 0 && atomicCAS(P.err + 1, 0, 7) == 0) {
                        atomicCAS(P.err, 0, MP_ERR_CHECK);
                        const int* l = (cur.goff >= 0) ? (arena1 + cur.goff) : (arena + (-cur.goff - 1));
                        double* d = P.dbg;
                        d[0] = cur.c1; d[1] = cur.len; d[2] = cur.maxr; d[3] = P.size[cur.c1];
                        d[4] = P.left[cur.c1]; d[5] = cur.goff; d[6] = arena_top; d[7] = sp;
                        d[8] = blk; d[9] = cur.mink;
                        for (int q = 0; q < 8 && q < cur.len; ++q) {
                            d[10 + 2 * q] = l[q];
                            d[11 + 2 * q] = sqrt(mp_dist_sq(P, cur.c1, l[q])) + P.size[l[q]];
                        }
                    }
                    break;
                }
                const int c1 = cur.c1;
                const double s1 = P.size[c1];
                // oneBinLessThan of each list's previous maximum
                const double thresh1_2 = (1. - P.binsize) * cur.maxr;
                const double thresh1_3 = THREE ? (1. - P.binsize) * cur.maxr3 : 0.;
                const int* list = (cur.goff >= 0) ? (arena1 + cur.goff) : nullptr;
                const int* list2 = (cur.goff < 0) ? (arena + (-cur.goff - 1)) : nullptr;
                const long long nbase = arena_top;
                double* S = slot_ptr(P, blk, cur.slot);
                if (tid < 2) max_sh[tid] = 0ull;
                double mymax = 0., mymax3 = 0.;
                float best = 0.f, best3 = 0.f;       // this thread's largest FP32 r + s, and its cell
                int bestc = -1, best3c = -1;
                int myany = 0, acc_n = 0, n_new = 0, parity = 0;
                bool full = false;
                const float4* c1t = reinterpret_cast<const float4*>(P.tc + c1);
                const float4 c1a = __ldg(c1t), c1b = __ldg(c1t + 1);
                const int left1 = __float_as_int(__ldg(c1t + 2).w);
                const float s1f = c1a.w;
                const float thresh1f_2 = (float)thresh1_2, thresh1f_3 = (float)thresh1_3;
                const int len = cur.len;
                for (int j0 = 0; j0 < len; j0 += MB) {
                    const int j = j0 + tid;
                    int cnt = 0, ca = -1, cb = -1, acc_ok = 0, kacc = -1;
                    double racc = 0., lracc = 0.;
                    const int c2 = j < len ? __ldcg(list ? list + j : list2 + j) : 0;
                    // A vertex-3 cell of a three-field cross: its own threshold, maximum and
                    // bins [nbd, 2 nbd).
                    const bool is3 = THREE && c2 >= P.base3;
                    const double thresh1 = is3 ? thresh1_3 : thresh1_2;
                    const float thresh1f = is3 ? thresh1f_3 : thresh1f_2;
                    bool dec32 = false;          // decided (and recorded) in FP32
                    float rs32 = 0.f;            // r + s of an FP32-decided unaccepted entry
                    float r32 = 0.f, lr32 = 0.f, dxf = 0.f, dyf = 0.f;
                    float4 ta, tb, tq, td;       // the packed cell c2
                    const bool inlist = j < cur.len && c2 >= 0 && c2 < P.ncells;
                    if (inlist) {
                        const float4* t4 = reinterpret_cast<const float4*>(P.tc + c2);
                        ta = __ldg(t4); tb = __ldg(t4 + 1); tq = __ldg(t4 + 2); td = __ldg(t4 + 3);
                    }
                    const bool valid = inlist && __float_as_int(tq.z) > 0;
                    if (j < cur.len && !valid) mp_check_fail(P.err, 2);
                    else if (j < cur.len) {
                        // Geometry from the hi/lo float positions, decisions in FP32.
                        const float s2f = ta.w;
                        dxf = (ta.x - c1a.x) + (tb.x - c1b.x);
                        dyf = (ta.y - c1a.y) + (tb.y - c1b.y);
                        float dsq = dxf * dxf + dyf * dyf;
                        if (P.coords != FLAT) {
                            const float dzf = (ta.z - c1a.z) + (tb.z - c1b.z);
                            dsq += dzf * dzf;
                        }
                        float rsqf = dsq;
                        if (P.metric == ARC) {
                            const float th = arc_from_chord_sq(dsq);
                            rsqf = th * th;
                        }
                        int k32 = -1;
                        bool sp1 = false, sp2 = false, any32 = false;
                        const int kind = mp_decide32(P, rsqf, s1f, s2f, thresh1f, k32, r32, lr32,
                                                     sp1, sp2, any32);
                        if (kind >= 0) {
                            dec32 = true;
                            if (kind == 1) {
                                acc_ok = 1; kacc = k32; ca = c2;
                            } else if (kind == 2) {
                                rs32 = r32 + (s1f + s2f);
                                if (any32) myany = 1;
                                if (sp2) { ca = __float_as_int(tq.w); cb = __float_as_int(td.x); cnt = 2; }
                                else { ca = c2; cnt = 1; }
                            }
                        }
                    }
                    if (j < cur.len && !dec32 && valid) {
                        const double s2 = P.size[c2];
                        const double rsq = mp_dist_sq(P, c1, c2);
                        const double s = s1 + s2;
                        if (!mp_too_small(P, rsq, s) && !mp_too_large(P, rsq, s)) {
                            int k = -1;
                            double r = sqrt(rsq), lr = 0.;
                            if (mp_single_bin(P, rsq, s, k, r, lr)) {
                                if (rsq >= P.minsepsq && rsq < P.maxsepsq) {
                                    if (k < 0) {
                                        lr = log(r);
                                        k = int((lr - P.logminsep) / P.binsize);
                                    }
                                    if (k >= P.nbd) k = P.nbd - 1;
                                    acc_ok = 1; kacc = k; racc = r; lracc = lr;
                                    ca = c2;
                                }
                            } else {
                                if (is3) mymax3 = fmax(mymax3, r + s);
                                else mymax = fmax(mymax, r + s);
                                // CalcSplitSq (include/Split.h:82-101)
                                double bsq_eff = rsq * fmin(P.bsq, P.asq);
                                bool split1, split2;
                                if (s2 > s1) {
                                    split2 = true;
                                    split1 = !(s2 > 2. * s1) && (s1 * s1 > 0.3422 * bsq_eff);
                                } else {
                                    split1 = true;
                                    split2 = !(s1 > 2. * s2) && (s2 * s2 > 0.3422 * bsq_eff);
                                }
                                if (split1 && r + s > thresh1) myany = 1;
                                if (split2) { ca = P.left[c2]; cb = P.right[c2]; cnt = 2; }
                                else { ca = c2; cnt = 1; }
                            }
                        }
                    }
                    // The maximum of r + s over the unaccepted entries is kept exact (it sets
                    // the next pass's thresholds).  A thread keeps its largest FP32 value; of
                    // two within the FP32 error of each other both get their FP64 value.  (FP64
                    // instructions take 16 cycles of the SM each: they are for the few entries
                    // that can be the maximum.)
                    if (rs32 > 0.f) {
                        float& bs = is3 ? best3 : best;
                        int& bc = is3 ? best3c : bestc;
                        if (rs32 > bs * (1.f + 1.6e-5f)) {
                            bs = rs32;
                            bc = c2;
                        } else if (rs32 > bs * (1.f - 1.6e-5f)) {
                            const double rs64 = sqrt(mp_dist_sq(P, c1, c2)) + (s1 + (double)ta.w);
                            if (is3) mymax3 = fmax(mymax3, rs64);
                            else mymax = fmax(mymax, rs64);
                            bs = fmaxf(bs, rs32);
                        }
                    }
                    if (acc_ok && is3) kacc += P.nbd;
                    // Places of the new entries and the accepted records (one barrier: the next
                    // chunk writes the other buffer).
                    const unsigned lt = (1u << lane) - 1u;
                    const unsigned b1 = __ballot_sync(0xffffffffu, cnt >= 1);
                    const unsigned b2 = __ballot_sync(0xffffffffu, cnt == 2);
                    const unsigned ba = __ballot_sync(0xffffffffu, acc_ok);
                    if (lane == 0) scan_sh[parity][wid] = make_int2(__popc(b1) + __popc(b2), __popc(ba));
                    __syncthreads();
                    int pos = __popc(b1 & lt) + __popc(b2 & lt), apos = __popc(ba & lt);
                    int tot_new = 0, tot_acc = 0;
#pragma unroll
                    for (int w = 0; w < MW; ++w) {
                        const int2 t = scan_sh[parity][w];
                        if (w < wid) { pos += t.x; apos += t.y; }
                        tot_new += t.x;
                        tot_acc += t.y;
                    }
                    parity ^= 1;
                    const long long wbase = nbase + n_new;
                    if (wbase + tot_new > P.arena2_cap || acc_n + tot_acc > P.acc_cap) {
                        if (tid == 0) set_mp_err(P.err, MP_ERR_ARENA);
                        full = true;
                    } else {
                        if (cnt >= 1) arena[wbase + pos] = ca;
                        if (cnt == 2) arena[wbase + pos + 1] = cb;
                        if (acc_ok && dec32 && P.coords == FLAT) {
                            // calculateGn's per-pair terms in FP32: ExpIPhi z = d / r, the
                            // spin-2 factor e = conj(d^2) / |d|^2, the projected shear wg and
                            // the scalar sums.
                            const float inv = __frcp_rn(r32 > 0.f ? r32 : 1.f);
                            float zr = dxf * inv, zi = dyf * inv;
                            // |z| = 1 again: r's rounding and its reciprocal's would come n-fold
                            // into z^n (rms error of z^12 9.0 u, with a division 7.7, so 5.2;
                            // u = 2^-24).
                            const float h = -0.5f * fmaf(zr, zr, fmaf(zi, zi, -1.f));
                            zr = fmaf(zr, h, zr);
                            zi = fmaf(zi, h, zi);
                            // (no rotation for the real payload of N / K pairs)
                            const bool rl = (P.pspin0 >> (is3 ? 1 : 0)) & 1;
                            const float er = rl ? 1.f : zr * zr - zi * zi;
                            const float ei = rl ? 0.f : -2.f * zr * zi;
                            const float w2 = tb.w;
                            const float4 lf = __ldg(P.lsf + ca);
                            const float l0 = lf.x, l1 = lf.y, l2 = lf.z, l3 = lf.w;
                            const float g1 = tq.x, g2 = tq.y;
                            const float wgr = g1 * er - g2 * ei, wgi = g1 * ei + g2 * er;
                            const float e2r = er * er - ei * ei, e2i = 2.f * er * ei;
                            const float wsr = l1 * e2r - l2 * e2i, wsi = l1 * e2i + l2 * e2r;
                            // z^2 in the self-pair sums of a spin-2 vertex; 1 for an N or K
                            // vertex (MultipoleScratch<GData>::calculateGn, buffer 0).
                            const float zsr = P.vreal ? 1.f : zr * zr - zi * zi;
                            const float zsi = P.vreal ? 0.f : 2.f * zr * zi;
                            const float a0r = wsr * zsr + wsi * zsi, a0i = wsi * zsr - wsr * zsi;
                            const float a1r = wsr * zsr - wsi * zsi, a1i = wsr * zsi + wsi * zsr;
                            float* R = acc + (size_t)(acc_n + apos) * MP_REC;
                            *reinterpret_cast<float4*>(R) = make_float4(zr, zi, wgr, wgi);
                            *reinterpret_cast<float4*>(R + 4) =
                                make_float4(w2, tq.z, __int_as_float(kacc), 0.f);
                            *reinterpret_cast<float4*>(R + 8) = make_float4(w2, w2 * r32, w2 * lr32, l0);
                            *reinterpret_cast<float4*>(R + 12) = make_float4(l0 * r32, l0 * lr32, a0r, a0i);
                            *reinterpret_cast<float4*>(R + 16) = make_float4(a1r, a1i, l3 * zsr, -l3 * zsi);
                            *reinterpret_cast<float4*>(R + 20) = make_float4(wgr, wgi, 0.f, 0.f);
                            atomicAdd(&bh[kacc], 1);
                        } else if (acc_ok) {
                            // The same terms from FP64 (non-flat geometry, or decided in FP64).
                            if (dec32) { racc = r32; lracc = lr32; }
                            C2 z, e;
                            phases(P, c1, ca, racc, z, e);
                            if ((P.pspin0 >> (is3 ? 1 : 0)) & 1) e = C2{1., 0.};
                            const double w2 = P.w[ca];
                            const double* ls = P.ls + 4 * (size_t)ca;
                            const C2 wg = cmul({(double)P.d1[ca], (double)P.d2[ca]}, e);
                            const C2 wgsq = cmul({ls[1], ls[2]}, cmul(e, e));
                            const C2 zsq = P.vreal ? C2{1., 0.} : cmul(z, z);
                            const C2 a0 = cmul(wgsq, conj2(zsq)), a1 = cmul(wgsq, zsq);
                            float* R = acc + (size_t)(acc_n + apos) * MP_REC;
                            *reinterpret_cast<float4*>(R) =
                                make_float4((float)z.re, (float)z.im, (float)wg.re, (float)wg.im);
                            *reinterpret_cast<float4*>(R + 4) =
                                make_float4((float)w2, __int_as_float(P.n[ca]), __int_as_float(kacc), 0.f);
                            *reinterpret_cast<float4*>(R + 8) =
                                make_float4((float)w2, (float)(w2 * racc), (float)(w2 * lracc), (float)ls[0]);
                            *reinterpret_cast<float4*>(R + 12) =
                                make_float4((float)(ls[0] * racc), (float)(ls[0] * lracc), (float)a0.re, (float)a0.im);
                            *reinterpret_cast<float4*>(R + 16) =
                                make_float4((float)a1.re, (float)a1.im, (float)(ls[3] * zsq.re), (float)(-ls[3] * zsq.im));
                            *reinterpret_cast<float4*>(R + 20) =
                                make_float4((float)wg.re, (float)wg.im, 0.f, 0.f);
                            atomicAdd(&bh[kacc], 1);
                        }
                    }
                    n_new += tot_new;
                    acc_n += tot_acc;
                    // (record buffer full, or the pass is over; the barrier also ends this
                    // chunk's writes to the list)
                    if (full) break;
                    const bool last = j0 + MB >= len;
                    if (last || acc_n > P.acc_cap - MB) {
                        __syncthreads();
                        if (acc_n > 0) mp_accumulate<H>(P, acc, perm, acc_n, S, bh, batches);
                        acc_n = 0;
                    }
                }
                // An overflow of the arenas leaves the lists incomplete: stop this job (the
                // call is retried with larger arenas).
                if (full) break;
                int mink = cur.mink;
                if (n_new == 0) {
                    zeta_emit(P, c1, S, 0, mink, out, diag, shG, shW, &zidx_sh, &job_emits);
                    break;
                }
                // The largest remaining separations: the threads whose FP32 value can be the
                // block's maximum take it in FP64.
                {
                    const unsigned any = __any_sync(0xffffffffu, myany) ? 0x80000000u : 0u;
                    const unsigned m2 = __reduce_max_sync(0xffffffffu, __float_as_uint(best));
                    const unsigned m3 = THREE ? __reduce_max_sync(0xffffffffu, __float_as_uint(best3)) : 0u;
                    if (lane == 0) { best_sh[0][wid] = m2 | any; best_sh[1][wid] = m3; }
                }
                __syncthreads();
                bool anysplit = false;
                {
                    unsigned bm2 = 0u, bm3 = 0u;
#pragma unroll
                    for (int w = 0; w < MW; ++w) {
                        const unsigned v = best_sh[0][w];
                        anysplit = anysplit || (v >> 31);
                        bm2 = max(bm2, v & 0x7fffffffu);
                        if (THREE) bm3 = max(bm3, best_sh[1][w]);
                    }
                    if (best > 0.f && best >= __uint_as_float(bm2) * (1.f - 8e-6f))
                        mymax = fmax(mymax, sqrt(mp_dist_sq(P, c1, bestc)) + (s1 + (double)P.size[bestc]));
                    if (mymax > 0.) atomicMax(&max_sh[0], (unsigned long long)__double_as_longlong(mymax));
                    if (THREE) {
                        if (best3 > 0.f && best3 >= __uint_as_float(bm3) * (1.f - 8e-6f))
                            mymax3 = fmax(mymax3, sqrt(mp_dist_sq(P, c1, best3c)) + (s1 + (double)P.size[best3c]));
                        if (mymax3 > 0.) atomicMax(&max_sh[1], (unsigned long long)__double_as_longlong(mymax3));
                    }
                }
                __syncthreads();
                const double maxrem2 = __longlong_as_double((long long)max_sh[0]);
                const double maxrem3 = THREE ? __longlong_as_double((long long)max_sh[1]) : 0.;
                const double maxrem = THREE ? fmax(maxrem2, maxrem3) : maxrem2;
                if (maxrem < P.maxsep) {
                    int k = 0;
                    if (!(maxrem < P.minsep)) {
                        // int((log(maxrem) - logminsep) / binsize) + 1, in FP64 only near an
                        // integer (FP32: 3e-7 of |log| + |logminsep|, over binsize).
                        const float lr = logf((float)maxrem);
                        const float kk = (lr - P.f_logminsep) / P.f_binsize;
                        const float err = 1e-5f * (1.f + fabsf(kk)) +
                                          1e-6f * (1.f + fabsf(lr) + fabsf(P.f_logminsep)) / P.f_binsize;
                        const float frac = kk - floorf(kk);
                        if (frac > err && frac < 1.f - err) k = (int)kk + 1;
                        else k = int((log(maxrem) - P.logminsep) / P.binsize) + 1;
                    }
                    if (k < mink) {
                        zeta_emit(P, c1, S, k, mink, out, diag, shG, shW, &zidx_sh, &job_emits);
                        mink = k;
                    }
                }
                const bool split1 = anysplit && left1 >= 0;
                if (tid == 0) {
                    arena_top = nbase + n_new;
                    alloc_ok = 1;
                    if (split1) {
                        if (free_cnt == 0 || sp + 1 > MSTACK) {
                            set_mp_err(P.err, MP_ERR_SLOTS);
                            alloc_ok = 0;
                        } else {
                            P2Entry rgt;
                            rgt.c1 = P.right[c1]; rgt.len = n_new; rgt.slot = free_list[--free_cnt];
                            rgt.mink = mink; rgt.goff = -nbase - 1;
                            rgt.maxr = maxrem2; rgt.maxr3 = maxrem3;
                            rgt.mark = nbase + n_new;
                            stk[sp++] = rgt;
                        }
                    }
                }
                __syncthreads();
                if (!alloc_ok) break;
                if (split1) {
                    // The right child gets a copy of the scratch (mp.duplicate()).
                    const double2* src = reinterpret_cast<const double2*>(S);
                    double2* dst = reinterpret_cast<double2*>(slot_ptr(P, blk, stk[sp - 1].slot));
                    const int half = (int)(P.slot_doubles / 2);
                    for (int q0 = tid; q0 < half; q0 += 8 * MB) {
                        double2 v[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) if (q0 + u * MB < half) v[u] = __ldcg(src + q0 + u * MB);
#pragma unroll
                        for (int u = 0; u < 8; ++u) if (q0 + u * MB < half) dst[q0 + u * MB] = v[u];
                    }
                }
                // Without a split, the old list is dead unless a pushed entry still uses it:
                // move the new list down onto it, so a chain of passes reuses one region.
                long long newoff = nbase;
                const bool old_in2 = cur.goff < 0;
                const long long oo = old_in2 ? (-cur.goff - 1) : 0;
                const bool old_used = (sp > 0 && stk[sp - 1].goff == cur.goff);
                if (!split1 && old_in2 && !old_used && oo < nbase) {
                    for (long long i0 = 0; i0 < n_new; i0 += MB) {
                        const long long i = i0 + tid;
                        int v = 0;
                        if (i < n_new) v = __ldcg(arena + nbase + i);
                        __syncthreads();
                        if (i < n_new) arena[oo + i] = v;
                        __syncthreads();
                    }
                    newoff = oo;
                }
                __syncthreads();
                if (tid == 0) {
                    if (split1) cur.c1 = left1;
                    cur.len = n_new;
                    cur.goff = -newoff - 1;
                    cur.mink = mink;
                    cur.maxr = maxrem2;
                    cur.maxr3 = maxrem3;
                    arena_top = newoff + n_new;
                }
                __syncthreads();
            }
            __syncthreads();
            if (tid == 0) free_list[free_cnt++] = cur.slot;
            __syncthreads();
        }
        // The largest record count of one job sizes the stop margin of later waves.
        if (tid == 0) atomicMax(P.zmaxjob, (unsigned long long)job_emits);
    }
}

// ---------------------------------------------------------------------------------------
static constexpr int ZB = 256;   // threads per block of the scalar sums
static constexpr int ZE = 2;     // entries per thread

// The n = 0 scalar outputs of calculateZeta over vertex records (ntri, meand2/3,
// meanlogd2/3): for every entry (a, b) whose min(a, b) lies in the record's rows,
//   a != b: ntri += n1 np_a np_b, meand2 += w1 sumw_b sumwr_a, meand3 += w1 sumw_a sumwr_b
//   a == b: ntri += n1 np_a (np_a - 1), meand2 = meand3 += w1 (sumw_a sumwr_a - sumwwr_a)
// (meanlogd likewise with sumwlogr).  ntri is an exact 64-bit integer sum; the means are FP32
// products with FP64 sums.  Block (g, tile) adds its sums to group g's partial arrays.
__global__ void __launch_bounds__(ZB) k_mp_zscal(ZParams Q, int chunk, double* spart,
                                                 unsigned long long* ntp)
{
    extern __shared__ float4 zsh[];    // [chunk][nb][2]
    __shared__ int4 hdr_sh[64];
    const int nb = Q.nbins;
    const int nb2 = nb * nb;
    const int g = blockIdx.x, tid = threadIdx.x;
    int ea[ZE], eb[ZE], em[ZE];     // entry (a, b) and min(a, b) mod nbd (the row mask)
    bool ev[ZE];
#pragma unroll
    for (int j = 0; j < ZE; ++j) {
        const int e = ((int)blockIdx.y * ZE + j) * ZB + tid;
        ev[j] = e < nb2;
        ea[j] = ev[j] ? e / nb : 0;
        eb[j] = ev[j] ? e % nb : 0;
        em[j] = min(ea[j] % Q.nbd, eb[j] % Q.nbd);
    }
    double D[ZE][4];
    unsigned long long C[ZE];
#pragma unroll
    for (int j = 0; j < ZE; ++j) { C[j] = 0ull; for (int q = 0; q < 4; ++q) D[j][q] = 0.; }
    const long long r0 = Q.nrec * g / gridDim.x, r1 = Q.nrec * (g + 1) / gridDim.x;
    for (long long c0 = r0; c0 < r1; c0 += chunk) {
        const int nv = (int)min((long long)chunk, r1 - c0);
        __syncthreads();
        for (int idx = tid; idx < nv * nb; idx += ZB) {
            const int v = idx / nb, a = idx % nb;
            const unsigned off = Q.off[c0 + v];
            if (off == ZOFF_NONE) {      // contracted in place
                if (a == 0) hdr_sh[v] = make_int4(0, 0, 0, 0);
                continue;
            }
            const float* R = Q.rec + 4 * (size_t)off;
            const float* RS = R + 8;
            float4* d = zsh + ((size_t)v * nb + a) * 2;
            d[0] = make_float4(RS[a], RS[nb + a], RS[2 * nb + a], RS[3 * nb + a]);
            d[1] = make_float4(RS[4 * nb + a], RS[5 * nb + a], 0.f, 0.f);
            if (a == 0)
                hdr_sh[v] = make_int4(__float_as_int(R[1]), __float_as_int(R[2]),
                                      __float_as_int(R[6]), __float_as_int(R[3]));
        }
        __syncthreads();
        float F[ZE][4];
#pragma unroll
        for (int j = 0; j < ZE; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) F[j][q] = 0.f;
        for (int v = 0; v < nv; ++v) {
            const int4 h = hdr_sh[v];
            const float w1 = __int_as_float(h.w);
            const unsigned long long n1 = (unsigned long long)h.z;
#pragma unroll
            for (int j = 0; j < ZE; ++j) {
                const int m = em[j];
                if (!ev[j] || m < h.x || m >= h.y) continue;
                const float4 pa = zsh[((size_t)v * nb + ea[j]) * 2];
                const unsigned long long npa = (unsigned)__float_as_int(pa.x);
                if (ea[j] == eb[j]) {
                    const float4 pa2 = zsh[((size_t)v * nb + ea[j]) * 2 + 1];
                    C[j] += n1 * npa * (npa > 0 ? npa - 1 : 0);
                    const float md = w1 * (pa.y * pa.z - pa2.x);
                    const float ml = w1 * (pa.y * pa.w - pa2.y);
                    F[j][0] += md; F[j][1] += ml; F[j][2] += md; F[j][3] += ml;
                } else {
                    const float4 pb = zsh[((size_t)v * nb + eb[j]) * 2];
                    C[j] += n1 * npa * (unsigned long long)(unsigned)__float_as_int(pb.x);
                    // (ordered = 1's meanlogd3 in the vertex-3 x vertex-2 block takes
                    // mp3.sumw at the column's bin, as the reference writes it)
                    const float swl = (Q.typo32 && ea[j] >= Q.nbd)
                        ? zsh[((size_t)v * nb + eb[j] % Q.nbd + Q.nbd) * 2].y : pa.y;
                    F[j][0] += w1 * pb.y * pa.z; F[j][1] += w1 * pb.y * pa.w;
                    F[j][2] += w1 * pa.y * pb.z; F[j][3] += w1 * swl * pb.w;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < ZE; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) D[j][q] += F[j][q];
    }
#pragma unroll
    for (int j = 0; j < ZE; ++j) {
        if (!ev[j]) continue;
        const int e = ea[j] * nb + eb[j];
#pragma unroll
        for (int q = 0; q < 4; ++q) spart[((size_t)g * 4 + q) * nb2 + e] += D[j][q];
        ntp[(size_t)g * nb2 + e] += C[j];
    }
}

// Final sums: what was contracted in place, the contraction's sums and the diagonal
// corrections.
__global__ void k_mp_reduce(int nblk, long long Z, int nb, int nn,
                            const double* in, const double* diag, long long diag_stride,
                            const double* part, int nsg, const double* spart,
                            const unsigned long long* ntp, double* out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 15 * Z) return;
    const int q = (int)(i / Z);
    const long long r = i % Z;
    double s = in[i];
    const int qp = q < 8 ? q : (q == 12 ? 8 : (q == 13 ? 9 : -1));
    const long long ab = r / nn;
    const int a = (int)(ab / nb), b = (int)(ab % nb), n = (int)(r % nn) - nn / 2;
    // The contraction's sums (zeta.cu: 4 x 2 tiles, n >= 0); those of (a, b, -n) are those of
    // (b, a, n) with gam2 and gam3 exchanged.  W_a conj(W_a) is real.
    if (qp >= 0 && !(a == b && qp == 9)) {
        const int ea = n < 0 ? b : a, eb = n < 0 ? a : b, an = n < 0 ? -n : n;
        const int qe = n < 0 && qp >= 4 && qp < 8 ? qp ^ 2 : qp;
        const int tcols = (nb + 1) >> 1, ntile = ((nb + 3) >> 2) * tcols;
        const int e = 2 * (ea & 3) + (eb & 1), tile = (ea >> 2) * tcols + (eb >> 1);
        s += part[((size_t)an * 80 + qe * 8 + e) * ntile + tile];
    }
    if (r % nn == nn / 2 && ((q >= 8 && q <= 11) || q == 14)) {
        const size_t nb2 = (size_t)nb * nb;
        if (q == 14) {
            unsigned long long c = 0ull;
            for (int g = 0; g < nsg; ++g) c += ntp[(size_t)g * nb2 + ab];
            s += (double)c;
        } else {
            for (int g = 0; g < nsg; ++g) s += spart[((size_t)g * 4 + (q - 8)) * nb2 + ab];
        }
    }
    if (a == b && (q < 8 || q == 12)) {
        const int d = q < 8 ? q : 8;
        for (int bl = 0; bl < nblk; ++bl) s -= diag[(size_t)bl * diag_stride + (size_t)d * nb + a];
    }
    out[i] = s;
}

// ---------------------------------------------------------------------------------------
// Host orchestration.

size_t mp_slot_doubles(int nb, int M)
{ return (2 * (size_t)nb * (M + 1) + 2 * (size_t)nb * (2 * M + 3) + 13 * (size_t)nb + 1) & ~(size_t)1; }

// 16-byte units of a vertex record of all bins
static long long mp_rec_units(int nb, int M)
{ return (8 + 2 * (long long)nb * (2 * M + 3) + 2 * nb * (M + 1) + 6 * nb + 3) / 4; }

int run_multipole(MPParams& P, MPScratch& X, int ntop, cudaStream_t st, double* h_out)
{
    const int nb = P.nbins, M = P.maxn, nn = 2 * M + 1;
    const long long Z = (long long)nb * nb * nn;
    int dev = 0, nsm = 0;
    TC_CU(cudaGetDevice(&dev));
    TC_CU(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const size_t inplace = sizeof(double) * (2 * (size_t)nb * (2 * M + 3) + 2 * (size_t)nb * (M + 1));
    const size_t shbytes = std::max(inplace, sizeof(AccBatch) * MW);
    if (inplace > 160 * 1024 || M + 1 > 64 || nb > MP_MAXNB) {
        set_last_error("the GPU multipole path needs max_n <= 63, nbins <= 128 and "
                       "nbins * max_n within its shared-memory staging");
        return 3;
    }
    // (powers up to 32, or up to 64 in two rounds)
    auto* kfin = M + 1 <= 32 ? (P.three ? k_mp_finish<true, 1> : k_mp_finish<false, 1>)
                             : (P.three ? k_mp_finish<true, 2> : k_mp_finish<false, 2>);
    TC_TRY(allow_smem(kfin, shbytes));
    int per = 0;
    TC_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kfin, MB, shbytes));
    if (per < 1) per = 1;
    const int nblk = nsm * std::min(per, MBLK);
    P.slot_doubles = (long long)mp_slot_doubles(nb, M);
    P.out_stride = 15 * Z;
    const int etiles = (nb * nb + ZE * ZB - 1) / (ZE * ZB);
    // Scalar outputs: records per chunk and record groups.
    const int chunk2 = (int)std::max<long long>(1, std::min<long long>(64, (48 * 1024) / (32LL * nb)));
    const size_t zsh2 = (size_t)chunk2 * nb * 32;
    // (with its static header array this can pass the 48 KB that needs no opt-in)
    TC_TRY(allow_smem(k_mp_zscal, zsh2));
    const int nsg = std::max(1, 2 * nsm / etiles);
    const long long recu = mp_rec_units(nb, M);
    const long long acc_cap = 4096;
    X.want_a1 = std::max<long long>(X.want_a1, 4LL * std::max(ntop, P.ntop2) + (1 << 16));
    X.want_jobs = std::max<long long>(X.want_jobs, 1 << 18);
    X.want_a2 = std::max<long long>(X.want_a2, 1 << 20);
    X.want_slots = std::max(X.want_slots, 32);
    for (int attempt = 0; attempt < 4; ++attempt) {
        // Allocate what is requested (the requests grow after an overflow).
        if (X.arena1_cap < X.want_a1 || (long long)ntop > X.ntop_alloc) {
            dfree(X.arena1);
            X.arena1_cap = 0;
            TC_TRY(dalloc(&X.arena1, (size_t)X.want_a1 * ntop));
            X.arena1_cap = X.want_a1; X.ntop_alloc = ntop;
        }
        if (X.jobs_cap < X.want_jobs) {
            dfree(X.jobs);
            X.jobs_cap = 0;
            TC_TRY(dalloc(&X.jobs, (size_t)X.want_jobs));
            X.jobs_cap = X.want_jobs;
        }
        const bool grow_blk = nblk > X.nblk;
        if (X.arena2_cap < X.want_a2 || grow_blk) {
            dfree(X.arena2);
            X.arena2_cap = 0;
            TC_TRY(dalloc(&X.arena2, (size_t)X.want_a2 * nblk));
            X.arena2_cap = X.want_a2;
        }
        if (X.acc_cap < acc_cap || grow_blk) {
            dfree(X.acc); dfree(X.perm);
            X.acc_cap = 0;
            TC_TRY(dalloc(&X.acc, (size_t)MP_REC * acc_cap * nblk));
            TC_TRY(dalloc(&X.perm, (size_t)acc_cap * nblk));
            X.acc_cap = acc_cap;
        }
        if (X.nslots < X.want_slots || grow_blk || P.slot_doubles != X.slot_doubles) {
            dfree(X.slots);
            X.nslots = 0;
            TC_TRY(dalloc(&X.slots, (size_t)X.want_slots * P.slot_doubles * nblk));
            X.nslots = X.want_slots; X.slot_doubles = P.slot_doubles;
        }
        if (grow_blk || P.out_stride > X.out_stride || 9LL * nb > X.diag_stride) {
            dfree(X.out); dfree(X.total); dfree(X.diag);
            X.out_stride = 0; X.diag_stride = 0;
            TC_TRY(dalloc(&X.out, (size_t)P.out_stride));
            TC_TRY(dalloc(&X.total, (size_t)P.out_stride));
            TC_TRY(dalloc(&X.diag, (size_t)9 * nb * nblk));
            X.out_stride = P.out_stride; X.diag_stride = 9LL * nb;
        }
        {
            // The vertex-record buffer: up to 32 GiB and a quarter of the free memory, or the
            // byte count in TCGPU_MP_RECORD_BYTES (at least 16 records of all bins).  With one
            // buffer for all records there is one wave: each wave ends with the blocks' last
            // jobs (10 ms of 240 at 500,000 points, 17 GB of records).  A cell leaves three
            // records or so, and the stop margin below is for the blocks' jobs in flight.
            size_t budget = (size_t)32 << 30;
            if (const char* ev = std::getenv("TCGPU_MP_RECORD_BYTES"))
                budget = std::min<size_t>((size_t)48 << 30, (size_t)std::max(0LL, std::atoll(ev)));   // (32-bit offsets)
            const long long want = (16LL * P.ncells + (1 << 19)) * recu;
            const long long cap = std::max<long long>(16 * recu, std::min<long long>((long long)(budget / 16), want));
            if (!X.zrec || X.zrec_units != recu || X.zcap < cap || (X.zcap > cap && cap < want)) {
                dfree(X.zrec); dfree(X.zoff); dfree(X.order);
                X.zcap = 0;
                size_t fr = 0, tot = 0;
                TC_CU(cudaMemGetInfo(&fr, &tot));
                X.zcap = 0;
                const long long c2 = std::min(cap, std::max<long long>(16 * recu, (long long)(fr / 4 / 16)));
                // (records hold the bins from ks on: room for numbers of half the size)
                X.zmax = 2 * c2 / recu + 16;
                TC_TRY(dalloc(&X.zrec, 4 * (size_t)c2));
                TC_TRY(dalloc(&X.zoff, (size_t)X.zmax));
                TC_TRY(dalloc(&X.order, (size_t)X.zmax));
                X.zcap = c2; X.zrec_units = recu;
            }
        }
        if (X.nsg < nsg || X.spart_nb2 < (long long)nb * nb) {
            dfree(X.spart); dfree(X.ntp);
            X.nsg = 0;
            TC_TRY(dalloc(&X.spart, (size_t)nsg * 4 * nb * nb));
            TC_TRY(dalloc(&X.ntp, (size_t)nsg * nb * nb));
            X.nsg = nsg; X.spart_nb2 = (long long)nb * nb;
        }
        const size_t npart = zeta_part_doubles(nb, M);
        if (X.npart < npart) {
            dfree(X.part);
            X.npart = 0;
            TC_TRY(dalloc(&X.part, npart));
            X.npart = npart;
        }
        const long long nkey = (long long)P.nbd * (P.nbd + 1), nsegs = zeta_segments(X.zmax, nb, P.nbd);
        if (X.nkey < nkey || X.nsegs < nsegs) {
            dfree(X.keys); dfree(X.segs);
            X.nkey = 0; X.nsegs = 0;
            TC_TRY(dalloc(&X.keys, 2 * (size_t)nkey + 2));
            TC_TRY(dalloc(&X.segs, (size_t)nsegs));
            X.nkey = nkey; X.nsegs = nsegs;
        }
        if (!X.ctl) TC_TRY(dalloc(&X.ctl, 4));
        if (!X.err) TC_TRY(dalloc(&X.err, 2));
        if (!X.dbg) TC_TRY(dalloc(&X.dbg, 32));
        X.nblk = std::max(X.nblk, nblk);
        P.arena1 = X.arena1; P.arena1_cap = X.arena1_cap;
        P.jobs = X.jobs; P.jobs_cap = X.jobs_cap;
        P.njobs = X.ctl; P.job_next = X.ctl + 1; P.zcount = X.ctl + 2; P.zmaxjob = X.ctl + 3;
        P.arena2 = X.arena2; P.arena2_cap = X.arena2_cap;
        P.acc = X.acc; P.perm = X.perm; P.acc_cap = (int)X.acc_cap;
        P.slots = X.slots; P.nslots = X.nslots;
        P.out = X.out;
        P.diag = X.diag;
        P.zrec = X.zrec; P.zcap = X.zcap; P.zoff = X.zoff; P.zmax = X.zmax;
        // Jobs are not started once the buffer is nearly full; the blocks' jobs in flight then
        // add at most nblk x (the largest job so far) records.
        auto set_zstop = [&](long long maxjob) {
            const long long margin = (long long)nblk * std::max<long long>(64, 2 * maxjob);
            P.zstop = std::max<long long>(X.zcap / 4, X.zcap - margin * recu);
            P.zmaxstop = std::max<long long>(X.zmax / 4, X.zmax - margin);
        };
        set_zstop(512);
        P.err = X.err;
        P.dbg = X.dbg;
        TC_CU(cudaMemsetAsync(X.ctl, 0, 4 * sizeof(unsigned long long), st));
        X.overflow = 0; X.records = 0; X.waves = 0;
        TC_CU(cudaMemsetAsync(X.err, 0, 2 * sizeof(int), st));
        TC_CU(cudaMemsetAsync(X.out, 0, sizeof(double) * (size_t)P.out_stride, st));
        TC_CU(cudaMemsetAsync(X.diag, 0, sizeof(double) * (size_t)9 * nb * nblk, st));
        TC_CU(cudaMemsetAsync(X.part, 0, sizeof(double) * npart, st));
        TC_CU(cudaMemsetAsync(X.spart, 0, sizeof(double) * (size_t)nsg * 4 * nb * nb, st));
        TC_CU(cudaMemsetAsync(X.ntp, 0, sizeof(unsigned long long) * (size_t)nsg * nb * nb, st));
        count_launch();
        k_mp_split1<<<ntop, MB, 0, st>>>(P);
        TC_CU(cudaGetLastError());
        unsigned long long nj = 0;
        int e = 0;
        TC_CU(cudaMemcpyAsync(&nj, X.ctl, sizeof(nj), cudaMemcpyDeviceToHost, st));
        TC_CU(cudaMemcpyAsync(&e, X.err, sizeof(int), cudaMemcpyDeviceToHost, st));
        TC_CU(cudaStreamSynchronize(st));
        P.njobs_val = (long long)nj;
        // Waves: the finish kernel runs jobs until the record buffer is nearly full, then the
        // records are contracted and the buffer is reused.
        for (int wave = 0; e == 0; ++wave) {
            TC_CU(cudaMemsetAsync(X.ctl + 2, 0, sizeof(unsigned long long), st));
            count_launch();
            kfin<<<nblk, MB, shbytes, st>>>(P);
            TC_CU(cudaGetLastError());
            unsigned long long c[4] = {0, 0, 0, 0};
            TC_CU(cudaMemcpyAsync(c, X.ctl, sizeof(c), cudaMemcpyDeviceToHost, st));
            TC_CU(cudaMemcpyAsync(&e, X.err, sizeof(int), cudaMemcpyDeviceToHost, st));
            TC_CU(cudaStreamSynchronize(st));
            if (e) break;
            ZParams Q;
            const long long emitted = (long long)(c[2] / ZC_ONE);
            Q.rec = X.zrec; Q.off = X.zoff; Q.nrec = std::min<long long>(emitted, X.zmax);
            Q.nbins = nb; Q.maxn = M;
            Q.part = X.part; Q.order = X.order; Q.segs = X.segs;
            Q.count = X.keys; Q.first = X.keys + X.nkey; Q.nseg = X.keys + 2 * X.nkey + 1;
            Q.shift = P.vreal ? 0 : 1;
            Q.nbd = P.nbd; Q.typo32 = P.typo32;
            if (Q.nrec > 0) {
                TC_TRY(launch_zeta(Q, nsm, st));
                if (!P.quick) {
                    count_launch();
                    k_mp_zscal<<<dim3(nsg, etiles), ZB, zsh2, st>>>(Q, chunk2, X.spart, X.ntp);
                    TC_CU(cudaGetLastError());
                }
            }
            // (contracted in place: those without a number, and those whose units did not fit)
            int placed = 0;
            TC_CU(cudaMemcpyAsync(&placed, Q.first + nkey, sizeof(int), cudaMemcpyDeviceToHost, st));
            TC_CU(cudaStreamSynchronize(st));
            X.overflow += emitted - (Q.nrec > 0 ? placed : 0);
            X.records += emitted;
            ++X.waves;
            set_zstop((long long)c[3]);
            if ((long long)c[1] >= P.njobs_val) break;
            if (wave > (1 << 24)) { e = MP_ERR_STACK; break; }
        }
        if (e == MP_ERR_ARENA || e == MP_ERR_JOBS || e == MP_ERR_SLOTS) {
            X.want_a1 = X.arena1_cap * 4; X.want_jobs = X.jobs_cap * 4;
            X.want_a2 = X.arena2_cap * 4;
            X.want_slots = std::min(X.nslots * 2, 64);
            continue;
        }
        if (e == MP_ERR_CHECK) {
            int site = 0;
            double d[32];
            TC_CU(cudaMemcpy(&site, X.err + 1, sizeof(int), cudaMemcpyDeviceToHost));
            TC_CU(cudaMemcpy(d, X.dbg, sizeof(d), cudaMemcpyDeviceToHost));
            std::string msg = "multipole: internal consistency check failed at site " +
                              std::to_string(site);
            if (site == 4 || site == 7) {
                msg += " [";
                for (int q = 0; q < 26; ++q) msg += std::to_string(d[q]) + " ";
                msg += "]";
            }
            set_last_error(msg);
            return 4;
        }
        if (e) {
            set_last_error("multipole: device stack overflow (tree too deep)");
            return 4;
        }
        count_launch();
        k_mp_reduce<<<(unsigned)((P.out_stride + 255) / 256), 256, 0, st>>>(
            nblk, Z, nb, nn, X.out, X.diag, 9LL * nb, X.part,
            P.quick ? 0 : nsg, X.spart, X.ntp, X.total);
        TC_CU(cudaGetLastError());
        TC_CU(cudaMemcpyAsync(h_out, X.total, sizeof(double) * (size_t)P.out_stride,
                              cudaMemcpyDeviceToHost, st));
        TC_CU(cudaStreamSynchronize(st));
        return 0;
    }
    set_last_error("multipole scratch still too small after retries");
    return 4;
}

void free_mp_scratch(MPScratch& X)
{
    dfree(X.arena1); dfree(X.jobs); dfree(X.arena2); dfree(X.acc); dfree(X.perm);
    dfree(X.slots); dfree(X.out); dfree(X.diag); dfree(X.total); dfree(X.zrec); dfree(X.part);
    dfree(X.spart); dfree(X.ntp);
    dfree(X.ctl); dfree(X.err); dfree(X.dbg);
    dfree(X.order); dfree(X.keys); dfree(X.segs); dfree(X.zoff);
    X = MPScratch();
}

}  // namespace tc
