// tree_build.cu -- GPU ball-tree build with the reference's cell rules.
//
// The tree is the one TreeCorr builds (src/Field.cpp:27-81 SetupTopLevelCells,
// src/Cell.cpp:556-615 BuildCell, src/Cell.cpp:426-554 SplitData): every cell holds the
// wpos-weighted centroid of its points (normalised on the sphere), the float sum of w,
// the float payload sum (parallel-transported to the centroid on the sphere), and
// size = float(max |centroid - p|); it is split at the centroid coordinate (Mean) or the
// bounding-box middle (Middle) along the axis of largest extent, while size^2 > min_size^2.
// The top-level phase splits regardless of min_size until size <= max_size and min_top
// levels are done, or max_top levels are reached.
//
// GB300 layout: the build is level-synchronous.  Cells with more than SMALL points are
// processed cooperatively by many blocks (chunks of CH points, deterministic two-stage FP64
// reductions, a stable scatter into the other of two point buffers); a level's tasks are
// written by the level before, so that no level waits for the host.  Cells with at most SMALL
// points (fewer for small catalogs) are finished by one block each, which keeps the points in shared memory
// and builds the whole subtree on them.
// Cell ids are positional, so no allocation counter is needed: an internal cell that
// splits [s,e) at m gets id m-1, a leaf starting at point s gets id (n-1)+s.
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdio>
#include <vector>
#include <algorithm>

#include "tc_internal.cuh"
#include "tc_host.hpp"
#include "traverse2pt.hpp"

namespace tc {

// ---------------------------------------------------------------------------------------
// device helpers

__device__ __forceinline__ void set_err(int* err, int code)
{ atomicCAS(err, 0, code); }

// a / n for several a: one division, then Markstein's correction of a * (1 / n), which gives
// the correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34, 1990) for operands
// without over- or underflow; other quotients (0, infinities, NaN, tiny or huge values) take
// the division itself.
struct Divisor {
    double n, inv;
    bool plain;
    __device__ __forceinline__ explicit Divisor(double n_) : n(n_), inv(1. / n_)
    { const double a = fabs(n_); plain = a > 1e-100 && a < 1e100; }
    __device__ __forceinline__ double operator()(double a) const
    {
        const double b = fabs(a);
        if (!(plain && b > 1e-100 && b < 1e100)) return a / n;
        const double q = a * inv;
        return fma(fma(-q, n, a), inv, q);
    }
};

// Position<Sphere>::normalize, include/Position.h:258-263.
__device__ __forceinline__ void normalize3(double& x, double& y, double& z)
{
    double n = sqrt(x * x + y * y + z * z);
    if (n == 0.) { x = 1.; y = 0.; z = 0.; }
    else {
        const Divisor by(n);
        x = by(x); y = by(y); z = by(z);
    }
}

// Bounds::getSplit, include/Bounds.h:65-66 (Flat) and 133-141 (ThreeD/Sphere).
__device__ __forceinline__ int split_axis(int coords, double xr, double yr, double zr)
{
    if (coords == FLAT) return yr > xr ? 1 : 0;
    return yr > xr ? (zr > yr ? 2 : 1) : (zr > xr ? 2 : 0);
}

// One point's contribution to the parallel-transported sum of a spin-s value,
// src/Cell.cpp:276-321.  (cx,cy,cz) is the centre as Position<Sphere> (normalised for
// ThreeD), cz_raw its raw z.
__device__ __forceinline__ void transport_add(int coords, int spin, double cx, double cy,
                                              double cz, double cz_raw, double px, double py,
                                              double pz, double wr, double wi, double& sr,
                                              double& si)
{
    if (spin == 0) { sr += wr; si += wi; return; }   // calculate_expmsialpha<0> = 1
    if (coords == THREED) normalize3(px, py, pz);
    double dsq = (cx - px) * (cx - px) + (cy - py) * (cy - py) + (cz - pz) * (cz - pz);
    if (dsq < 1.e-12) { sr += wr; si += wi; return; }
    double z1 = cz_raw, z2 = pz;
    double cosA = (z1 - z2) + 0.5 * z2 * dsq;
    double sinA = cy * px - cx * py;
    double cosB = (z2 - z1) + 0.5 * z1 * dsq;
    double sinB = sinA;
    double cb = -cosA * cosB + sinA * sinB;
    double sb = sinA * cosB + cosA * sinB;
    // calculate_expmsialpha<s>(cb + i sb), include/ProjectHelper.h:33-60.
    double er, ei;
    if (spin == 2) {
        double nrm = cb * cb + sb * sb;
        if (!(nrm > 0.)) nrm = 1.;
        er = (cb * cb - sb * sb) / nrm;
        ei = -(2. * cb * sb) / nrm;
    } else if (spin == 1) {
        double nrm = cb * cb + sb * sb;
        if (!(nrm > 0.)) nrm = 1.;
        nrm = sqrt(nrm);
        er = cb / nrm;
        ei = -sb / nrm;
    } else if (spin == 3) {
        // r^3, then conj(r^3) / |r^3|.
        const double r2r = cb * cb - sb * sb, r2i = 2. * cb * sb;
        const double r3r = r2r * cb - r2i * sb, r3i = r2r * sb + r2i * cb;
        double nrm = r3r * r3r + r3i * r3i;
        if (!(nrm > 0.)) nrm = 1.;
        nrm = sqrt(nrm);
        er = r3r / nrm;
        ei = -r3i / nrm;
    } else {
        // r^2 squared, then conj(r^4) / |r^2|^2.
        const double r2r = cb * cb - sb * sb, r2i = 2. * cb * sb;
        const double r4r = r2r * r2r - r2i * r2i, r4i = 2. * r2r * r2i;
        double nrm = r2r * r2r + r2i * r2i;
        if (!(nrm > 0.)) nrm = 1.;
        er = r4r / nrm;
        ei = -r4i / nrm;
    }
    sr += wr * er - wi * ei;
    si += wr * ei + wi * er;
}

// Writes a finished cell and links it to its parent.
__device__ __forceinline__ void write_cell(const Cells& C, int id, double x, double y, double z,
                                           float size, float w, float d1, float d2, int n,
                                           int s, int parent, int side)
{
    C.x[id] = x; C.y[id] = y; C.z[id] = z;
    C.size[id] = size; C.w[id] = w; C.d1[id] = d1; C.d2[id] = d2;
    C.n[id] = n; C.start[id] = s;
    C.left[id] = -1; C.right[id] = -1;
    C.parent[id] = parent;
    if (parent >= 0) {
        if (side == 0) C.left[parent] = id;
        else C.right[parent] = id;
    }
}

__device__ __forceinline__ void add_top(int* tops, int* ntop, int id, int s)
{
    int k = atomicAdd(ntop, 1);
    tops[2 * k] = s;
    tops[2 * k + 1] = id;
}

// The decision of SetupTopLevelCells (src/Field.cpp:57-80) followed by BuildCell
// (src/Cell.cpp:595-613).  Returns true to split.  Updates the task's top-phase state.
__device__ __forceinline__ bool decide_split(const BuildParams& P, int& intop, int mintop,
                                             int maxtop, double sizesq, bool& is_top)
{
    is_top = false;
    if (intop) {
        if (sizesq == 0. || (sizesq <= P.maxsizesq && mintop <= 0) || maxtop <= 0) {
            is_top = true;
            intop = 0;
        } else {
            return true;   // top-level phase: split regardless of min_size
        }
    }
    return sizesq > P.minsizesq;
}

__device__ __forceinline__ float cell_size(const BuildParams& P, double sizesq)
{ return P.brute ? __int_as_float(0x7f800000) : float(sqrt(sizesq)); }

// Copies point i of buffer A into slot j of buffer B.
__device__ __forceinline__ void move_point(const Points& A, int i, const Points& B, int j)
{
    B.x[j] = A.x[i]; B.y[j] = A.y[i]; B.z[j] = A.z[i]; B.wp[j] = A.wp[i];
    B.w[j] = A.w[i]; B.d1[j] = A.d1[i]; B.d2[j] = A.d2[i]; B.idx[j] = A.idx[i];
}

// ---------------------------------------------------------------------------------------
// Input preparation: Field::Field copies every point into a CellData (src/Field.cpp:180-196);
// Position<Sphere> normalises (include/Position.h:245), w is stored as float, and the
// payload as float(w*k) or complex<float>(w*g) (include/Cell.h:138-140, 176-178).

__global__ void k_prepare(int n, int coords, int dkind, const double* x, const double* y,
                          const double* z, const double* d1, const double* d2, const double* w,
                          const double* wpos, Points P)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double px = x[i], py = y[i], pz = (z && coords != FLAT) ? z[i] : 0.;
    if (coords == SPHERE) normalize3(px, py, pz);
    double wi = w[i];
    P.x[i] = px; P.y[i] = py; P.z[i] = pz;
    P.wp[i] = wpos ? wpos[i] : wi;
    P.w[i] = float(wi);
    if (dkind == DK) { P.d1[i] = float(wi * d1[i]); P.d2[i] = 0.f; }
    else if (dkind == DG) { P.d1[i] = float(wi * d1[i]); P.d2[i] = float(wi * d2[i]); }
    else { P.d1[i] = 0.f; P.d2[i] = 0.f; }
    P.idx[i] = i;
}

// ---------------------------------------------------------------------------------------
// Deterministic warp reductions (butterflies).

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_min(double v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_isum(int v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Doubles as integers of the same order: a comparison is two ALU instructions, where FP64
// comparisons share the FP64 pipe (1/64 of the FP32 rate) that bounds the build.
__device__ __forceinline__ long long dkey(double v)
{
    const long long b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double dunkey(long long k)
{ return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL)); }

__device__ __forceinline__ long long warp_kmin(long long v)
{
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ long long warp_kmax(long long v)
{
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sums v[0..N) over the warp by a reduce-scatter (N <= 8, half of the values travel per
// step) and hands every lane all totals: 9 FP64 adds per lane for five values where five
// butterflies take 25.
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N], int lane)
{
    static_assert(N <= 8, "");
    double a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = q < N ? v[q] : 0.;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const int half = 4 >> s, o = 16 >> s;
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < half; ++q) {
            if (q >= N) continue;                      // both partners hold zeros
            const double send = up ? a[q] : a[q + half];
            const double keep = up ? a[q + half] : a[q];
            a[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    // Lane bits 4, 3, 2 picked the upper half at each step: value q sits at lanes 4 q.
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = __shfl_sync(0xffffffffu, a[0], 4 * q);
}

// transport_add for a point at squared distance dsq from the centre; the spin-2 phase takes
// one reciprocal for its two divisions.
__device__ __forceinline__ void transport_near(int coords, int spin, double cx, double cy,
                                               double cz, double cz_raw, double px, double py,
                                               double pz, double dsq, double wr, double wi,
                                               double& sr, double& si)
{
    if (spin != 2 || coords == THREED) {
        transport_add(coords, spin, cx, cy, cz, cz_raw, px, py, pz, wr, wi, sr, si);
        return;
    }
    if (dsq < 1.e-12) { sr += wr; si += wi; return; }
    const double cosA = (cz - pz) + 0.5 * pz * dsq;
    const double sinA = cy * px - cx * py;
    const double cosB = (pz - cz) + 0.5 * cz * dsq;
    const double cb = -cosA * cosB + sinA * sinA;
    const double sb = sinA * cosB + cosA * sinA;
    double nrm = cb * cb + sb * sb;
    if (!(nrm > 0.)) nrm = 1.;
    const double inv = 1. / nrm;
    const double er = (cb * cb - sb * sb) * inv;
    const double ei = -(2. * cb * sb) * inv;
    sr += wr * er - wi * ei;
    si += wr * ei + wi * er;
}

// ---------------------------------------------------------------------------------------
// Cooperative levels (cells with more than SMALL points).

// The root [0, n) as level 0's task.
__global__ void k_level_root(LevelBufs L, BuildTask root)
{
    const int n = root.e - root.s, nc = (n + L.ch - 1) / L.ch;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c == 0) {
        L.tasks[0][0] = root;
        L.tchunk[0][0] = make_int2(0, nc);
        L.cnt[0] = make_int2(1, nc);
    }
    if (c < nc) {
        Chunk k;
        k.task = 0; k.cs = root.s + c * L.ch; k.ce = min(k.cs + L.ch, root.e);
        k.leftoff = k.rightoff = 0;
        L.chunks[0][c] = k;
    }
}

// Counts a chunk of task t as done; true for the whole block of the task's last one, whose
// first warp then reads all its chunks' partials (with __ldcg: other blocks wrote them).
__device__ __forceinline__ bool task_complete(const LevelBufs& L, int t, int nchunk, int* flag)
{
    if (threadIdx.x == 0) {
        __threadfence();
        const int k = atomicAdd(&L.done[t], 1);
        *flag = k == nchunk - 1;
        if (*flag) L.done[t] = 0;
    }
    __syncthreads();
    const bool last = *flag != 0;
    if (last) __threadfence();
    return last;
}

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }

// One warp: centroid, weight, split axis and value of task t.
__device__ void task_combine1(const LevelBufs& L, int lev, int t, Points P0, Points P1, const BuildParams& BP)
{
    const int lane = threadIdx.x & 31;
    const int2 tc = L.tchunk[lev & 1][t];
    const int c0 = tc.x, c1 = tc.x + tc.y;
    double s[5] = {0., 0., 0., 0., 0.};
    double xmin = DBL_MAX, ymin = DBL_MAX, zmin = DBL_MAX;
    double xmax = -DBL_MAX, ymax = -DBL_MAX, zmax = -DBL_MAX;
    for (int c = c0 + lane; c < c1; c += 32) {
        const Part1* p = L.part1 + c;
        s[0] += ldcg(&p->sx); s[1] += ldcg(&p->sy); s[2] += ldcg(&p->sz);
        s[3] += ldcg(&p->swp); s[4] += ldcg(&p->sw);
        xmin = fmin(xmin, ldcg(&p->xmin)); xmax = fmax(xmax, ldcg(&p->xmax));
        ymin = fmin(ymin, ldcg(&p->ymin)); ymax = fmax(ymax, ldcg(&p->ymax));
        zmin = fmin(zmin, ldcg(&p->zmin)); zmax = fmax(zmax, ldcg(&p->zmax));
    }
    warp_sums<5>(s, lane);
    xmin = dunkey(warp_kmin(dkey(xmin))); xmax = dunkey(warp_kmax(dkey(xmax)));
    ymin = dunkey(warp_kmin(dkey(ymin))); ymax = dunkey(warp_kmax(dkey(ymax)));
    zmin = dunkey(warp_kmin(dkey(zmin))); zmax = dunkey(warp_kmax(dkey(zmax)));
    if (lane) return;
    const BuildTask tk = L.tasks[lev & 1][t];
    const Points& P = tk.buf ? P1 : P0;
    TaskStats r;
    // BuildCellData, src/Cell.cpp:170-200.
    if (s[3] != 0.) {
        r.cx = s[0] / s[3]; r.cy = s[1] / s[3]; r.cz = s[2] / s[3];
        if (BP.coords == SPHERE) normalize3(r.cx, r.cy, r.cz);
    } else {
        r.cx = P.x[tk.s]; r.cy = P.y[tk.s]; r.cz = P.z[tk.s];
    }
    r.w = float(s[4]);
    r.axis = split_axis(BP.coords, xmax - xmin, ymax - ymin, zmax - zmin);
    if (BP.split == MIDDLE) {   // Bounds::getMiddle, include/Bounds.h:67-68
        r.splitval = r.axis == 2 ? (zmax + zmin) / 2. : r.axis == 1 ? (ymax + ymin) / 2.
                                                                     : (xmax + xmin) / 2.;
    } else {                    // Mean: the centroid, src/Cell.cpp:481-495
        r.splitval = r.axis == 2 ? r.cz : r.axis == 1 ? r.cy : r.cx;
    }
    // Remember whether all points share the split coordinate (needed by the fallback).
    double lo = r.axis == 2 ? zmin : r.axis == 1 ? ymin : xmin;
    double hi = r.axis == 2 ? zmax : r.axis == 1 ? ymax : xmax;
    r.allsame = (lo == hi) ? 1 : 0;
    r.mid = -1;
    r.copy = 0;
    r.byindex = 0;
    r.sizesq = 0.;
    L.stats[t] = r;
}

__global__ void __launch_bounds__(CB) k_chunk_pass1(LevelBufs L, int lev, Points P0, Points P1, BuildParams BP)
{
    after_previous();
    __shared__ double sh[CB / 32][5];
    __shared__ long long shk[CB / 32][6];
    __shared__ int flag;
    if ((int)blockIdx.x >= L.cnt[lev].y) return;
    const Chunk ch = L.chunks[lev & 1][blockIdx.x];
    const Points& P = L.tasks[lev & 1][ch.task].buf ? P1 : P0;
    double s[5] = {0., 0., 0., 0., 0.};
    long long k[6];                       // minima and, negated, maxima
    const long long big = dkey(DBL_MAX);
#pragma unroll
    for (int q = 0; q < 3; ++q) { k[2 * q] = big; k[2 * q + 1] = ~dkey(-DBL_MAX); }
    const bool flat = BP.coords == FLAT;
    if (flat) { k[4] = 0; k[5] = ~0ll; }
#pragma unroll 4
    for (int i = ch.cs + threadIdx.x; i < ch.ce; i += CB) {
        const double px = P.x[i], py = P.y[i], wp = P.wp[i];
        s[0] += px * wp; s[1] += py * wp; s[3] += wp; s[4] += P.w[i];
        const long long kx = dkey(px), ky = dkey(py);
        k[0] = min(k[0], kx); k[1] = min(k[1], ~kx);
        k[2] = min(k[2], ky); k[3] = min(k[3], ~ky);
        if (!flat) {
            const double pz = P.z[i];
            s[2] += pz * wp;
            const long long kz = dkey(pz);
            k[4] = min(k[4], kz); k[5] = min(k[5], ~kz);
        }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    warp_sums<5>(s, lane);
#pragma unroll
    for (int q = 0; q < 6; ++q) k[q] = warp_kmin(k[q]);
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 5; ++q) sh[wid][q] = s[q];
#pragma unroll
        for (int q = 0; q < 6; ++q) shk[wid][q] = k[q];
    }
    __syncthreads();
    // Thread q combines quantity q over the warps, in their order.
    if (threadIdx.x < 5) {
        double t = 0.;
        for (int w = 0; w < CB / 32; ++w) t += sh[w][threadIdx.x];
        sh[0][threadIdx.x] = t;
    } else if (threadIdx.x >= 32 && threadIdx.x < 38) {
        long long t = shk[0][threadIdx.x - 32];
        for (int w = 1; w < CB / 32; ++w) t = min(t, shk[w][threadIdx.x - 32]);
        shk[0][threadIdx.x - 32] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        Part1 r;
        r.sx = sh[0][0]; r.sy = sh[0][1]; r.sz = sh[0][2]; r.swp = sh[0][3]; r.sw = sh[0][4];
        r.xmin = dunkey(shk[0][0]); r.xmax = dunkey(~shk[0][1]);
        r.ymin = dunkey(shk[0][2]); r.ymax = dunkey(~shk[0][3]);
        r.zmin = dunkey(shk[0][4]); r.zmax = dunkey(~shk[0][5]);
        L.part1[blockIdx.x] = r;
    }
    if (task_complete(L, ch.task, L.tchunk[lev & 1][ch.task].y, &flag) && threadIdx.x < 32)
        task_combine1(L, lev, ch.task, P0, P1, BP);
}

// One warp: finishes task t's cell, decides, sets the scatter offsets of its chunks and appends
// the children to the next level or to the small cells.
__device__ void task_combine2(const LevelBufs& L, int lev, int t, const BuildParams& BP, const Cells& C,
                              int* tops, int* ntop, int* err)
{
    const int lane = threadIdx.x & 31;
    const BuildTask tk = L.tasks[lev & 1][t];
    const int2 tc = L.tchunk[lev & 1][t];
    TaskStats s = L.stats[t];
    Chunk* chunks = L.chunks[lev & 1] + tc.x;
    const Part2* part = L.part2 + tc.x;
    long long ks = dkey(0.);
    double pp[2] = {0., 0.};
    int nleft = 0;
    for (int c = lane; c < tc.y; c += 32) {
        ks = max(ks, dkey(ldcg(&part[c].sizesq)));
        pp[0] += ldcg(&part[c].pr); pp[1] += ldcg(&part[c].pi);
        nleft += __ldcg(&part[c].nleft);
    }
    const double sizesq = dunkey(warp_kmax(ks));
    warp_sums<2>(pp, lane);
    nleft = warp_isum(nleft);
    const int n = tk.e - tk.s;
    bool is_top;
    int intop = tk.intop;
    bool split = decide_split(BP, intop, tk.mintop, tk.maxtop, sizesq, is_top);
    int mid = tk.s + nleft;
    int byindex = 0;
    bool handed = false;
    if (split && (nleft == 0 || nleft == n)) {
        // SplitData falls back to Median when the mean puts everything on one side
        // (src/Cell.cpp:526-551).  On a cooperative level this is only done when every
        // point shares the split coordinate, where any order is a valid nth_element; other
        // cells of at most SMALL points go to k_subtree as they are, which ranks the points.
        if (s.allsame) { mid = (tk.s + tk.e) / 2; byindex = 1; }
        else if (n <= SMALL) { handed = true; split = false; }
        else { if (lane == 0) set_err(err, DEV_DEGENERATE_SPLIT); split = false; }
    }
    float d1 = float(pp[0]), d2 = float(pp[1]);
    if (BP.dkind == DN) { d1 = 0.f; d2 = 0.f; }
    if (BP.dkind == DK) d2 = 0.f;
    const int id = split ? mid - 1 : (BP.n - 1) + tk.s;
    if (lane == 0) {
        if (handed) {
            L.small[atomicAdd(L.nsmall, 1)] = tk;
        } else {
            write_cell(C, id, s.cx, s.cy, s.cz, split ? cell_size(BP, sizesq) : 0.f, s.w, d1, d2, n,
                       tk.s, tk.parent, tk.side);
            if (is_top) add_top(tops, ntop, id, tk.s);
        }
        s.mid = split ? mid : -1;
        s.copy = (!split && !handed && tk.buf == 1) ? 1 : 0;
        s.byindex = byindex;
        L.stats[t] = s;
    }
    if (!split) return;
    // Chunk offsets for the stable scatter.
    int loff = 0, roff = 0;
    for (int b = 0; b < tc.y; b += 32) {
        const int c = b + lane;
        int nl = 0, len = 0;
        if (c < tc.y) {
            const int cs = chunks[c].cs, ce = chunks[c].ce;
            nl = byindex ? max(0, min(ce, mid) - cs) : __ldcg(&part[c].nleft);
            len = ce - cs;
        }
        int xl = nl, xa = len;
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, xl, o), e = __shfl_up_sync(0xffffffffu, xa, o);
            if (lane >= o) { xl += a; xa += e; }
        }
        if (c < tc.y) {
            chunks[c].leftoff = loff + xl - nl;
            chunks[c].rightoff = roff + (xa - xl) - (len - nl);
        }
        const int tl = __shfl_sync(0xffffffffu, xl, 31), ta = __shfl_sync(0xffffffffu, xa, 31);
        loff += tl;
        roff += ta - tl;
    }
    for (int k = 0; k < 2; ++k) {
        BuildTask c = tk;
        if (k == 0) c.e = mid;
        else c.s = mid;
        c.parent = id;
        c.side = k;
        c.intop = intop;
        c.mintop = tk.mintop - 1;
        c.maxtop = tk.maxtop - 1;
        c.buf = tk.buf ^ 1;
        const int m = c.e - c.s;
        if (m <= L.sub) {
            if (lane == 0) L.small[atomicAdd(L.nsmall, 1)] = c;
            continue;
        }
        const int nc = (m + L.ch - 1) / L.ch;
        int at = 0, first = 0;
        if (lane == 0) {
            at = atomicAdd(&L.cnt[lev + 1].x, 1);
            first = atomicAdd(&L.cnt[lev + 1].y, nc);
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (at >= L.cap_tasks || first + nc > L.cap_chunks) {      // (sized for any split)
            if (lane == 0) set_err(err, DEV_TASK_OVERFLOW);
            return;
        }
        if (lane == 0) {
            L.tasks[(lev + 1) & 1][at] = c;
            L.tchunk[(lev + 1) & 1][at] = make_int2(first, nc);
        }
        for (int q = lane; q < nc; q += 32) {
            Chunk w;
            w.task = at; w.cs = c.s + q * L.ch; w.ce = min(w.cs + L.ch, c.e);
            w.leftoff = w.rightoff = 0;
            L.chunks[(lev + 1) & 1][first + q] = w;
        }
    }
}

// center != 0: only the largest distance from the centroid, into stats (field_center).
__global__ void __launch_bounds__(CB) k_chunk_pass2(LevelBufs L, int lev, Points P0, Points P1,
                                                     BuildParams BP, Cells C, int* tops, int* ntop,
                                                     int* err, int center)
{
    after_previous();
    __shared__ double sh[CB / 32][3];
    __shared__ int shi[CB / 32];
    __shared__ int flag;
    if ((int)blockIdx.x >= L.cnt[lev].y) return;
    const Chunk ch = L.chunks[lev & 1][blockIdx.x];
    const TaskStats s = L.stats[ch.task];
    const Points& P = L.tasks[lev & 1][ch.task].buf ? P1 : P0;
    const int coords = BP.coords, dkind = center ? DN : BP.dkind, spin = BP.spin;
    double cx = s.cx, cy = s.cy, cz = s.cz;
    double tcx = cx, tcy = cy, tcz = cz;
    if (coords == THREED) normalize3(tcx, tcy, tcz);
    long long ks = dkey(0.);
    const long long ksplit = dkey(s.splitval);
    const bool splits0 = 0. < s.splitval;
    double pr = 0., pi = 0.;
    int nleft = 0;
    for (int i = ch.cs + threadIdx.x; i < ch.ce; i += CB) {
        double px = P.x[i], py = P.y[i], pz = P.z[i];
        double d = (cx - px) * (cx - px) + (cy - py) * (cy - py);
        if (coords != FLAT) d += (cz - pz) * (cz - pz);
        ks = max(ks, dkey(d));
        double c = s.axis == 2 ? pz : s.axis == 1 ? py : px;
        // (0 and -0 are equal, their keys are not)
        nleft += ((__double_as_longlong(c) << 1) == 0 ? splits0 : dkey(c) < ksplit) ? 1 : 0;
        if (dkind == DK) {
            pr += P.d1[i];
        } else if (dkind == DG) {
            if (coords == FLAT) { pr += P.d1[i]; pi += P.d2[i]; }
            else transport_near(coords, spin, tcx, tcy, tcz, cz, px, py, pz, d, P.d1[i], P.d2[i], pr, pi);
        }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double sizesq = dunkey(warp_kmax(ks));
    double pp[2] = {pr, pi};
    if (dkind != DN) warp_sums<2>(pp, lane);
    nleft = warp_isum(nleft);
    if (lane == 0) { sh[wid][0] = sizesq; sh[wid][1] = pp[0]; sh[wid][2] = pp[1]; shi[wid] = nleft; }
    __syncthreads();
    if (threadIdx.x == 0) {
        Part2 r;
        r.sizesq = 0.; r.pr = 0.; r.pi = 0.;
        r.nleft = 0; r.pad = 0;
        for (int w = 0; w < CB / 32; ++w) {
            r.sizesq = fmax(r.sizesq, sh[w][0]);
            r.pr += sh[w][1]; r.pi += sh[w][2];
            r.nleft += shi[w];
        }
        L.part2[blockIdx.x] = r;
    }
    const int2 tc = L.tchunk[lev & 1][ch.task];
    if (!task_complete(L, ch.task, tc.y, &flag) || threadIdx.x >= 32) return;
    if (!center) {
        task_combine2(L, lev, ch.task, BP, C, tops, ntop, err);
        return;
    }
    long long m = dkey(0.);
    for (int c = lane; c < tc.y; c += 32) m = max(m, dkey(ldcg(&L.part2[tc.x + c].sizesq)));
    m = warp_kmax(m);
    if (lane == 0) L.stats[ch.task].sizesq = dunkey(m);
}

// Stable partition of each split chunk into the other buffer (or a copy of a leaf's
// points into buffer 0).
__global__ void __launch_bounds__(CB) k_chunk_scatter(LevelBufs L, int lev, Points P0, Points P1)
{
    after_previous();
    __shared__ int wsum[2][CB / 32];
    if ((int)blockIdx.x >= L.cnt[lev].y) return;
    const Chunk ch = L.chunks[lev & 1][blockIdx.x];
    const BuildTask tk = L.tasks[lev & 1][ch.task];
    const TaskStats s = L.stats[ch.task];
    const Points& A = tk.buf ? P1 : P0;
    const Points& B = tk.buf ? P0 : P1;
    if (s.mid < 0) {
        if (s.copy) for (int i = ch.cs + threadIdx.x; i < ch.ce; i += CB) move_point(A, i, P0, i);
        return;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool by_index = s.byindex != 0;
    int lbase = tk.s + ch.leftoff;
    int rbase = s.mid + ch.rightoff;
    for (int base = ch.cs; base < ch.ce; base += CB) {
        int i = base + threadIdx.x;
        bool valid = i < ch.ce;
        bool left = false;
        if (valid) {
            if (by_index) left = i < s.mid;
            else {
                double c = s.axis == 2 ? A.z[i] : s.axis == 1 ? A.y[i] : A.x[i];
                left = c < s.splitval;
            }
        }
        unsigned bl = __ballot_sync(0xffffffffu, valid && left);
        unsigned br = __ballot_sync(0xffffffffu, valid && !left);
        unsigned lt = (1u << lane) - 1u;
        if (lane == 0) { wsum[0][wid] = __popc(bl); wsum[1][wid] = __popc(br); }
        __syncthreads();
        int lpre = 0, rpre = 0, ltot = 0, rtot = 0;
        for (int k = 0; k < CB / 32; ++k) {
            if (k < wid) { lpre += wsum[0][k]; rpre += wsum[1][k]; }
            ltot += wsum[0][k]; rtot += wsum[1][k];
        }
        if (valid) {
            int dst = left ? lbase + lpre + __popc(bl & lt) : rbase + rpre + __popc(br & lt);
            move_point(A, i, B, dst);
        }
        lbase += ltot;
        rbase += rtot;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// Block-finished subtrees (cells with at most SMALL points).

__device__ __forceinline__ int pack_meta(int side, int intop, int buf, int mintop, int maxtop)
{
    mintop = max(-2000, min(2000, mintop)) + 2048;
    maxtop = max(-2000, min(2000, maxtop)) + 2048;
    return side | (intop << 1) | (buf << 2) | (mintop << 8) | (maxtop << 20);
}

// Cells of at most thread_t points (THREAD_T or THREAD_FEW) are finished by one thread, sums in
// point order.  Small cells are ~94% of a subtree's cells, and a warp spends the same
// reductions on a 2-point cell as on a 2048-point one.
constexpr int THREAD_T = 32;
// Catalogs whose subtrees hold at most FEW_SUB points leave each SM one or two of them, and the
// chain of one thread's points is what a block waits for: there warps go on down to THREAD_FEW
// points.  Whole builds of spin-2 points on the sphere, 32 -> 12: 5000 points 0.67 -> 0.62 ms, 25,000
// 0.75 -> 0.71 (8 and 16 within 2% of 12); at 100,000 points, with FEW_SUB 512, 8 took 1.09
// against 1.03, so the line lies below.  Blocks above FEW_N points keep THREAD_T.
constexpr int THREAD_FEW = 12, FEW_N = 512, FEW_SUB = 256;
constexpr int SB = 256;             // threads of a subtree block
constexpr int SW = SB / 32;
constexpr unsigned NOT_SINGLE = ~0u;
constexpr int SBIG = SMALL / (THREAD_T + 1) + 1;   // cells above THREAD_T points at one depth
static_assert(FEW_N / (THREAD_FEW + 1) < SBIG, "a depth's cells fit its list");

// One subtree's points, in shared memory for the whole build of the subtree: the points stay
// where they are and the cells permute 16-bit indices, so a level moves 2 bytes per point
// instead of 48.
struct SubPoints {
    double x[SMALL], y[SMALL], z[SMALL], wp[SMALL];
    float w[SMALL], d1[SMALL], d2[SMALL];
    unsigned short perm[2][SMALL];
    unsigned single[SMALL];         // position of a one-point cell: (parent + 1, index buffer,
                                    // side) packed, or NOT_SINGLE
};
struct SubPart {                    // one warp's share of a cell that several warps work on
    double sum[5];                  // x wp, y wp, z wp, wp, w
    long long lo[3], hi[3];         // bounds as ordered keys
    double sizesq, pr, pi;
    int nleft;
};
struct SubCentre {
    double cx, cy, cz, tcx, tcy, tcz, splitval;
    int axis;
};
struct SubShared {
    SubPoints P;
    WTask cell[2][SBIG];            // cells above thread_t points of this and the next depth
    int ncell[2], nsmall[2];
    SubPart part[SW];
    SubCentre centre[SW];
};

// The first pass over the points i0, i0 + step, .. < e of a cell: sums and bounds.
template <bool FLATC>
__device__ __forceinline__ void sub_pass1(const SubPoints& P, const unsigned short* perm, int i0,
                                          int e, int step, double (&s)[5], long long (&lo)[3],
                                          long long (&hi)[3])
{
#pragma unroll
    for (int q = 0; q < 5; ++q) s[q] = 0.;
#pragma unroll
    for (int q = 0; q < 3; ++q) { lo[q] = dkey(DBL_MAX); hi[q] = dkey(-DBL_MAX); }
    if (FLATC) { lo[2] = 0; hi[2] = 0; }
    for (int i = i0; i < e; i += step) {
        const int p = perm[i];
        const double px = P.x[p], py = P.y[p], wp = P.wp[p];
        s[0] += px * wp; s[1] += py * wp; s[3] += wp; s[4] += P.w[p];
        const long long kx = dkey(px), ky = dkey(py);
        lo[0] = min(lo[0], kx); hi[0] = max(hi[0], kx);
        lo[1] = min(lo[1], ky); hi[1] = max(hi[1], ky);
        if (!FLATC) {
            const double pz = P.z[p];
            s[2] += pz * wp;
            const long long kz = dkey(pz);
            lo[2] = min(lo[2], kz); hi[2] = max(hi[2], kz);
        }
    }
}

// Centroid, split axis and value of a cell from its sums (src/Cell.cpp:170-200, 481-525).
template <bool FLATC>
__device__ __forceinline__ SubCentre sub_centre(const SubPoints& P, int first,
                                                const BuildParams& BP, const double (&s)[5],
                                                const long long (&lo)[3], const long long (&hi)[3])
{
    SubCentre c;
    if (s[3] != 0.) {
        const Divisor by(s[3]);
        c.cx = by(s[0]); c.cy = by(s[1]); c.cz = FLATC ? 0. : by(s[2]);
        if (!FLATC && BP.coords == SPHERE) normalize3(c.cx, c.cy, c.cz);
    } else {
        c.cx = P.x[first]; c.cy = P.y[first]; c.cz = FLATC ? 0. : P.z[first];
    }
    double l[3], h[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) { l[q] = dunkey(lo[q]); h[q] = dunkey(hi[q]); }
    c.axis = split_axis(FLATC ? FLAT : BP.coords, h[0] - l[0], h[1] - l[1], h[2] - l[2]);
    if (BP.split == MIDDLE)
        c.splitval = c.axis == 2 ? (h[2] + l[2]) / 2. : c.axis == 1 ? (h[1] + l[1]) / 2.
                                                                     : (h[0] + l[0]) / 2.;
    else
        c.splitval = c.axis == 2 ? c.cz : c.axis == 1 ? c.cy : c.cx;
    c.tcx = c.cx; c.tcy = c.cy; c.tcz = c.cz;
    if (!FLATC && BP.coords == THREED) normalize3(c.tcx, c.tcy, c.tcz);
    return c;
}

// The second pass: size, payload, points left of the split value.
template <bool FLATC, bool CPLX>
__device__ __forceinline__ void sub_pass2(const SubPoints& P, const unsigned short* perm, int i0,
                                          int e, int step, const BuildParams& BP,
                                          const SubCentre& c, double& sizesq, double& pr,
                                          double& pi, int& nleft)
{
    sizesq = 0.; pr = 0.; pi = 0.;
    nleft = 0;
    const double* ax = c.axis == 2 ? P.z : c.axis == 1 ? P.y : P.x;
    for (int i = i0; i < e; i += step) {
        const int p = perm[i];
        const double px = P.x[p], py = P.y[p], pz = FLATC ? 0. : P.z[p];
        double d = (c.cx - px) * (c.cx - px) + (c.cy - py) * (c.cy - py);
        if (!FLATC) d += (c.cz - pz) * (c.cz - pz);
        sizesq = fmax(sizesq, d);
        nleft += (ax[p] < c.splitval) ? 1 : 0;
        if (CPLX) {
            if (FLATC) { pr += P.d1[p]; pi += P.d2[p]; }
            else transport_near(BP.coords, BP.spin, c.tcx, c.tcy, c.tcz, c.cz, px, py, pz, d,
                                P.d1[p], P.d2[p], pr, pi);
        } else if (BP.dkind == DK) {
            pr += P.d1[p];
        }
    }
}

// Whether point i of [s, e) is among the mid - s smallest by (coordinate, position).
__device__ __forceinline__ bool sub_rank_left(const double* ax, const unsigned short* perm,
                                              int s, int e, int mid, int i)
{
    const double c = ax[perm[i]];
    int rank = 0;
    for (int j = s; j < e; ++j) {
        const double cj = ax[perm[j]];
        rank += (cj < c || (cj == c && j < i)) ? 1 : 0;
    }
    return rank < (mid - s);
}

// What follows the two passes of a cell: the decision, the split point and the cell itself
// (written by the caller's one thread).
struct SubSplit {
    bool split, rank;
    int mid, intop;
};
__device__ __forceinline__ SubSplit sub_finish(const BuildParams& BP, const WTask& w, int base,
                                               const SubCentre& c, float wsum, double sizesq,
                                               double pr, double pi, int nleft, bool writer,
                                               const Cells& C, int* tops, int* ntop)
{
    const int n = w.e - w.s;
    SubSplit r;
    r.intop = (w.meta >> 1) & 1;
    const int mintop = ((w.meta >> 8) & 0xfff) - 2048;
    const int maxtop = ((w.meta >> 20) & 0xfff) - 2048;
    bool is_top;
    r.split = decide_split(BP, r.intop, mintop, maxtop, sizesq, is_top);
    r.rank = (BP.split == MEDIAN);
    r.mid = w.s + nleft;
    if (r.split && !r.rank && (nleft == 0 || nleft == n)) r.rank = true;
    if (r.split && r.rank) r.mid = (w.s + w.e) / 2;   // SplitDataCore<Median>, src/Cell.cpp:464-479
    if (writer) {
        float d1 = float(pr), d2 = float(pi);
        if (BP.dkind == DN) { d1 = 0.f; d2 = 0.f; }
        if (BP.dkind == DK) d2 = 0.f;
        const int id = r.split ? base + r.mid - 1 : (BP.n - 1) + base + w.s;
        write_cell(C, id, c.cx, c.cy, c.cz, r.split ? cell_size(BP, sizesq) : 0.f, wsum, d1, d2,
                   n, base + w.s, w.parent, w.meta & 1);
        if (is_top) add_top(tops, ntop, id, base + w.s);
    }
    return r;
}

__device__ __forceinline__ WTask sub_child(const WTask& w, const SubSplit& r, int base, int side)
{
    const int mintop = ((w.meta >> 8) & 0xfff) - 2048;
    const int maxtop = ((w.meta >> 20) & 0xfff) - 2048;
    const int nb = ((w.meta >> 2) & 1) ^ 1;
    WTask c;
    c.s = side ? r.mid : w.s;
    c.e = side ? w.e : r.mid;
    c.parent = base + r.mid - 1;
    c.meta = pack_meta(side, r.intop, nb, mintop - 1, maxtop - 1);
    return c;
}

// A one-point child is noted at its position; the block writes these leaves together at the
// end, to consecutive ids.  (Ids of internal cells are below n < 2^30, so the packing holds.)
__device__ __forceinline__ void sub_single(SubPoints& P, const WTask& w, int base,
                                           const BuildParams& BP, int* tops, int* ntop)
{
    const int s = w.s, buf = (w.meta >> 2) & 1;
    P.single[s] = ((unsigned)(w.parent + 1) << 2) | (buf << 1) | (w.meta & 1);
    if ((w.meta >> 1) & 1) add_top(tops, ntop, (BP.n - 1) + base + s, base + s);
}

// A cell of 2 .. thread_t points by one thread.  Positions are relative to base (the block's
// first point); a finished cell's order ends up in perm[0].  Returns whether it was split,
// with its children in k.
template <bool FLATC, bool CPLX>
__device__ __forceinline__ bool sub_by_thread(const WTask& w, int base, SubPoints& P,
                                              const BuildParams& BP, const Cells& C, int* tops,
                                              int* ntop, WTask (&k)[2])
{
    const int s = w.s, e = w.e, buf = (w.meta >> 2) & 1;
    const unsigned short* perm = P.perm[buf];
    unsigned short* to = P.perm[buf ^ 1];
    double sum[5];
    long long lo[3], hi[3];
    sub_pass1<FLATC>(P, perm, s, e, 1, sum, lo, hi);
    const SubCentre c = sub_centre<FLATC>(P, perm[s], BP, sum, lo, hi);
    double sizesq, pr, pi;
    int nleft;
    sub_pass2<FLATC, CPLX>(P, perm, s, e, 1, BP, c, sizesq, pr, pi, nleft);
    const SubSplit r = sub_finish(BP, w, base, c, float(sum[4]), sizesq, pr, pi, nleft, true, C,
                                  tops, ntop);
    if (!r.split) {
        if (buf) for (int i = s; i < e; ++i) P.perm[0][i] = perm[i];
        return false;
    }
    // Stable partition into the other index buffer.
    const double* ax = c.axis == 2 ? P.z : c.axis == 1 ? P.y : P.x;
    int l = s, h = r.mid;
    for (int i = s; i < e; ++i) {
        const unsigned short p = perm[i];
        const bool left = r.rank ? sub_rank_left(ax, perm, s, e, r.mid, i) : ax[p] < c.splitval;
        const int dst = left ? l++ : h++;
        if (dst < e) to[dst] = p;
    }
    k[0] = sub_child(w, r, base, 0);
    k[1] = sub_child(w, r, base, 1);
    return true;
}

// A child of at most thread_t points: noted if it is one point, else onto the list.
__device__ __forceinline__ void sub_small(const WTask& k, int base, SubPoints& P,
                                          const BuildParams& BP, int* tops, int* ntop,
                                          WTask* list, int* count)
{
    if (k.e - k.s == 1) sub_single(P, k, base, BP, tops, ntop);
    else list[atomicAdd(count, 1)] = k;
}

// One warp's share (part of parts) of a cell above thread_t points; COOP: several warps of
// the block work on the cell and meet at block barriers (every warp of the block makes the
// same calls).  `on` is false for a warp without a cell in a COOP round.
template <bool FLATC, bool CPLX, bool COOP>
__device__ __forceinline__ void sub_cell(SubShared& S, bool on, WTask w, int part, int parts,
                                         int base, const BuildParams& BP, const Cells& C,
                                         int* tops, int* ntop, int next, WTask* small, int lane,
                                         int wid, int thread_t)
{
    SubPoints& P = S.P;
    const int n = w.e - w.s, buf = (w.meta >> 2) & 1;
    const unsigned short* perm = P.perm[buf];
    unsigned short* to = P.perm[buf ^ 1];
    const int per = ((n + parts - 1) / parts + 31) & ~31;
    const int i0 = min(w.e, w.s + part * per), i1 = min(w.e, i0 + per);
    const int p0 = wid - part;      // the first warp of this cell's group
    double sum[5];
    long long lo[3], hi[3];
    sub_pass1<FLATC>(P, perm, on ? i0 + lane : i1, i1, 32, sum, lo, hi);
    warp_sums<5>(sum, lane);
#pragma unroll
    for (int q = 0; q < (FLATC ? 2 : 3); ++q) { lo[q] = warp_kmin(lo[q]); hi[q] = warp_kmax(hi[q]); }
    if (COOP) {
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 5; ++q) S.part[wid].sum[q] = sum[q];
#pragma unroll
            for (int q = 0; q < 3; ++q) { S.part[wid].lo[q] = lo[q]; S.part[wid].hi[q] = hi[q]; }
        }
        __syncthreads();
        for (int t = 0; t < parts; ++t) {
            const SubPart& o = S.part[p0 + t];
#pragma unroll
            for (int q = 0; q < 5; ++q) sum[q] = t ? sum[q] + o.sum[q] : o.sum[q];
#pragma unroll
            for (int q = 0; q < 3; ++q) { lo[q] = min(lo[q], o.lo[q]); hi[q] = max(hi[q], o.hi[q]); }
        }
    }
    // One warp of the group: the FP64 pipe takes a warp's instruction in 16 cycles of the SM
    // (all warps computing it: 200,000 points 1.43 ms for the whole build, so 1.40).
    SubCentre c;
    if (COOP) {
        if (part == 0) {
            c = sub_centre<FLATC>(P, on ? perm[w.s] : 0, BP, sum, lo, hi);
            if (lane == 0) S.centre[wid] = c;
        }
        __syncthreads();
        c = S.centre[p0];
    } else {
        c = sub_centre<FLATC>(P, on ? perm[w.s] : 0, BP, sum, lo, hi);
    }
    double sizesq, pp[2];
    int nleft;
    sub_pass2<FLATC, CPLX>(P, perm, on ? i0 + lane : i1, i1, 32, BP, c, sizesq, pp[0], pp[1], nleft);
    sizesq = dunkey(warp_kmax(dkey(sizesq)));
    if (BP.dkind != DN) warp_sums<2>(pp, lane);
    nleft = warp_isum(nleft);
    int before = 0;                 // left points of the parts before this one
    if (COOP) {
        if (lane == 0) {
            SubPart& o = S.part[wid];
            o.sizesq = sizesq; o.pr = pp[0]; o.pi = pp[1]; o.nleft = nleft;
        }
        __syncthreads();
        nleft = 0;
        pp[0] = pp[1] = 0.;
        for (int t = 0; t < parts; ++t) {
            const SubPart& o = S.part[p0 + t];
            sizesq = fmax(sizesq, o.sizesq);
            pp[0] += o.pr; pp[1] += o.pi;
            if (t < part) before += o.nleft;
            nleft += o.nleft;
        }
    }
    if (on) {
        const SubSplit r = sub_finish(BP, w, base, c, float(sum[4]), sizesq, pp[0], pp[1], nleft,
                                      part == 0 && lane == 0, C, tops, ntop);
        if (!r.split) {
            if (buf) for (int i = i0 + lane; i < i1; i += 32) P.perm[0][i] = perm[i];
        } else {
            // Stable partition into the other index buffer.
            const double* ax = c.axis == 2 ? P.z : c.axis == 1 ? P.y : P.x;
            if (COOP && r.rank) {
                // By rank the parts before this one are counted anew.
                before = 0;
                for (int i = w.s + lane; i < i0; i += 32)
                    before += sub_rank_left(ax, perm, w.s, w.e, r.mid, i) ? 1 : 0;
                before = warp_isum(before);
            }
            int l = w.s + before, h = r.mid + (i0 - w.s) - before;
            const unsigned lt = (1u << lane) - 1u;
            for (int b = i0; b < i1; b += 32) {
                const int i = b + lane;
                const bool valid = i < i1;
                const unsigned short p = valid ? perm[i] : 0;
                bool left = false;
                if (valid) left = r.rank ? sub_rank_left(ax, perm, w.s, w.e, r.mid, i)
                                         : ax[p] < c.splitval;
                const unsigned bl = __ballot_sync(0xffffffffu, valid && left);
                const unsigned br = __ballot_sync(0xffffffffu, valid && !left);
                if (valid) {
                    const int dst = left ? l + __popc(bl & lt) : h + __popc(br & lt);
                    if (dst < w.e) to[dst] = p;
                }
                l += __popc(bl);
                h += __popc(br);
            }
            if (part == 0 && lane < 2) {
                const WTask k = sub_child(w, r, base, lane);
                if (k.e - k.s > thread_t) S.cell[next][atomicAdd(&S.ncell[next], 1)] = k;
                else sub_small(k, base, P, BP, tops, ntop, small, &S.nsmall[0]);
            }
        }
    }
}

// One block builds the whole subtree of a cell of at most SMALL points.  The points are read
// once into shared memory.  The cells above thread_t points are taken depth by depth, a few
// warps to a cell near the root, one further down; then the smaller ones in rounds, one
// thread to a cell and the children onto the next round's list, so that the lanes of a warp
// work on cells of like size (a thread that walked its own subtree would leave most lanes
// waiting: its cells of 2 points fall together with another lane's of 20).
// Bound: the FP64 pipe (2 lanes per clock and SM; ~50 FP64 instructions per point and depth
// with the parallel transport of a spin-2 field on the sphere, ~100 per cell) once the
// subtrees fill the chip, the chain of a subtree's depths for small catalogs.
// Measured, spin-2 field on the sphere, against one warp per subtree with the points in global
// memory: 10M points 42.8 -> 19.2 ms, 200K 6.8 -> 0.57 ms; 5000 flat points 2.7 -> 0.21 ms.
// A thread per cell of 32 points with its whole subtree took 34.0, 1.37 and 0.47 ms.
template <bool FLATC, bool CPLX>
__global__ void __launch_bounds__(SB, 2) k_subtree(const BuildTask* tasks, Points P0, Points P1,
                                                   BuildParams BP, Cells C, int* tops, int* ntop,
                                                   WTask* wstack, int thread_t, int* err)
{
    extern __shared__ __align__(16) unsigned char sub_sh[];
    SubShared& S = *reinterpret_cast<SubShared*>(sub_sh);
    SubPoints& P = S.P;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const BuildTask root = tasks[blockIdx.x];
    const int base = root.s, n = root.e - root.s;
    if (n > SMALL) {                        // (the host sends none)
        if (tid == 0) set_err(err, DEV_TASK_OVERFLOW);
        return;
    }
    if (n > FEW_N) thread_t = THREAD_T;
    // Lists of cells of 2 .. thread_t points, this round's and the next one's: the cells of a
    // list are disjoint, so n / 2 entries hold them.
    WTask* list[2] = {wstack + base, wstack + base + n / 2};
    const Points& A = root.buf ? P1 : P0;
    for (int i = tid; i < n; i += SB) {
        P.x[i] = A.x[base + i]; P.y[i] = A.y[base + i]; P.z[i] = A.z[base + i];
        P.wp[i] = A.wp[base + i];
        P.w[i] = A.w[base + i]; P.d1[i] = A.d1[base + i]; P.d2[i] = A.d2[base + i];
        P.perm[0][i] = P.perm[1][i] = (unsigned short)i;
        P.single[i] = NOT_SINGLE;
    }
    __syncthreads();
    if (tid == 0) {
        const WTask w = {0, n, root.parent, pack_meta(root.side, root.intop, 0, root.mintop, root.maxtop)};
        S.ncell[0] = S.ncell[1] = S.nsmall[0] = S.nsmall[1] = 0;
        if (n > thread_t) { S.cell[0][0] = w; S.ncell[0] = 1; }
        else sub_small(w, base, P, BP, tops, ntop, list[0], &S.nsmall[0]);
    }
    __syncthreads();
    // A depth's cells are disjoint and each holds more than thread_t points, so a list never
    // holds more than SBIG - 1 cells, and a cell has fewer points at every depth.
    for (int cur = 0;; cur ^= 1) {
        const int m = S.ncell[cur];
        if (m == 0) break;
        if (m * 2 <= SW) {
            const int parts = SW / (m == 1 ? 1 : m == 2 ? 2 : 4);
            const int ci = wid / parts;
            const bool on = ci < m;
            sub_cell<FLATC, CPLX, true>(S, on, S.cell[cur][on ? ci : 0], wid % parts, parts, base,
                                        BP, C, tops, ntop, cur ^ 1, list[0], lane, wid, thread_t);
        } else {
            for (int ci = wid; ci < m; ci += SW)
                sub_cell<FLATC, CPLX, false>(S, true, S.cell[cur][ci], 0, 1, base, BP, C, tops,
                                             ntop, cur ^ 1, list[0], lane, wid, thread_t);
        }
        __syncthreads();
        if (tid == 0) S.ncell[cur] = 0;
        __syncthreads();
    }
    for (int cur = 0;; cur ^= 1) {
        const int m = S.nsmall[cur];
        if (m == 0) break;
        for (int t = tid; t < m; t += SB) {
            WTask k[2];
            if (sub_by_thread<FLATC, CPLX>(list[cur][t], base, P, BP, C, tops, ntop, k)) {
                sub_small(k[0], base, P, BP, tops, ntop, list[cur ^ 1], &S.nsmall[cur ^ 1]);
                sub_small(k[1], base, P, BP, tops, ntop, list[cur ^ 1], &S.nsmall[cur ^ 1]);
            }
        }
        __syncthreads();
        if (tid == 0) S.nsmall[cur] = 0;
        __syncthreads();
    }
    // The points in tree order (the original indices read before any is overwritten) and the
    // one-point leaves (src/Cell.cpp:564-575).
    int idx[SMALL / SB], pos[SMALL / SB];
#pragma unroll
    for (int u = 0; u < SMALL / SB; ++u) {
        const int i = tid + u * SB;
        if (i >= n) continue;
        const unsigned sg = P.single[i];
        pos[u] = P.perm[sg != NOT_SINGLE ? (sg >> 1) & 1 : 0][i];
        idx[u] = A.idx[base + pos[u]];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < SMALL / SB; ++u) {
        const int i = tid + u * SB;
        if (i >= n) continue;
        const int p = pos[u];
        const double x = P.x[p], y = P.y[p], z = P.z[p];
        const float w = P.w[p], d1 = P.d1[p], d2 = P.d2[p];
        P0.x[base + i] = x; P0.y[base + i] = y; P0.z[base + i] = z;
        P0.wp[base + i] = P.wp[p];
        P0.w[base + i] = w; P0.d1[base + i] = d1; P0.d2[base + i] = d2;
        P0.idx[base + i] = idx[u];
        const unsigned sg = P.single[i];
        if (sg != NOT_SINGLE)
            write_cell(C, (BP.n - 1) + base + i, x, y, z, 0.f, w, d1, d2, 1, base + i,
                       (int)(sg >> 2) - 1, sg & 1);
    }
}

// Median splits of cells above SMALL points (rank by a count over the cell, which the
// cooperative levels have no pass for): one warp walks down from the root and leaves every
// cell of at most SMALL points to k_subtree.
__global__ void k_median_levels(BuildTask root, Points P0, Points P1, BuildParams BP, Cells C,
                                int* tops, int* ntop, WTask* stk, BuildTask* small_out,
                                int* nsmall_out, int* err)
{
    const int lane = threadIdx.x & 31;
    int sp = 0;
    if (lane == 0) {
        WTask w0 = {root.s, root.e, root.parent,
                    pack_meta(root.side, root.intop, root.buf, root.mintop, root.maxtop)};
        stk[0] = w0;
    }
    sp = 1;
    __syncwarp();
    while (sp > 0) {
        --sp;
        WTask w = stk[sp];
        __syncwarp();
        const int s = w.s, e = w.e, n = e - s;
        const int side = w.meta & 1, buf = (w.meta >> 2) & 1;
        int intop = (w.meta >> 1) & 1;
        const int mintop = ((w.meta >> 8) & 0xfff) - 2048;
        const int maxtop = ((w.meta >> 20) & 0xfff) - 2048;
        if (n <= SMALL) {
            if (lane == 0)
                small_out[atomicAdd(nsmall_out, 1)] =
                    BuildTask{s, e, w.parent, side, mintop, maxtop, intop, buf};
            continue;
        }
        const Points& A = buf ? P1 : P0;
        const Points& B = buf ? P0 : P1;
        // Pass 1: centroid, weight, bounds (src/Cell.cpp:170-200, 520-525).
        double sx = 0., sy = 0., sz = 0., swp = 0., sw = 0.;
        double xmin = DBL_MAX, ymin = DBL_MAX, zmin = DBL_MAX;
        double xmax = -DBL_MAX, ymax = -DBL_MAX, zmax = -DBL_MAX;
        for (int i = s + lane; i < e; i += 32) {
            double px = A.x[i], py = A.y[i], pz = A.z[i], wp = A.wp[i];
            sx += px * wp; sy += py * wp; sz += pz * wp; swp += wp; sw += A.w[i];
            xmin = fmin(xmin, px); xmax = fmax(xmax, px);
            ymin = fmin(ymin, py); ymax = fmax(ymax, py);
            zmin = fmin(zmin, pz); zmax = fmax(zmax, pz);
        }
        sx = warp_sum(sx); sy = warp_sum(sy); sz = warp_sum(sz); swp = warp_sum(swp);
        sw = warp_sum(sw);
        xmin = warp_min(xmin); ymin = warp_min(ymin); zmin = warp_min(zmin);
        xmax = warp_max(xmax); ymax = warp_max(ymax); zmax = warp_max(zmax);
        double cx, cy, cz;
        if (swp != 0.) {
            cx = sx / swp; cy = sy / swp; cz = sz / swp;
            if (BP.coords == SPHERE) normalize3(cx, cy, cz);
        } else {
            cx = A.x[s]; cy = A.y[s]; cz = A.z[s];
        }
        const int axis = split_axis(BP.coords, xmax - xmin, ymax - ymin, zmax - zmin);
        // Pass 2: size, payload.
        double tcx = cx, tcy = cy, tcz = cz;
        if (BP.coords == THREED) normalize3(tcx, tcy, tcz);
        double sizesq = 0., pr = 0., pi = 0.;
        for (int i = s + lane; i < e; i += 32) {
            double px = A.x[i], py = A.y[i], pz = A.z[i];
            double d = (cx - px) * (cx - px) + (cy - py) * (cy - py);
            if (BP.coords != FLAT) d += (cz - pz) * (cz - pz);
            sizesq = fmax(sizesq, d);
            if (BP.dkind == DK) pr += A.d1[i];
            else if (BP.dkind == DG) {
                if (BP.coords == FLAT) { pr += A.d1[i]; pi += A.d2[i]; }
                else transport_add(BP.coords, BP.spin, tcx, tcy, tcz, cz, px, py, pz, A.d1[i],
                                   A.d2[i], pr, pi);
            }
        }
        sizesq = warp_max(sizesq); pr = warp_sum(pr); pi = warp_sum(pi);
        bool is_top;
        const bool split = decide_split(BP, intop, mintop, maxtop, sizesq, is_top);
        const int mid = (s + e) / 2;    // SplitDataCore<Median>, src/Cell.cpp:464-479
        float d1 = float(pr), d2 = float(pi);
        if (BP.dkind == DN) { d1 = 0.f; d2 = 0.f; }
        if (BP.dkind == DK) d2 = 0.f;
        const int id = split ? mid - 1 : (BP.n - 1) + s;
        if (lane == 0) {
            write_cell(C, id, cx, cy, cz, split ? cell_size(BP, sizesq) : 0.f, float(sw), d1, d2,
                       n, s, w.parent, side);
            if (is_top) add_top(tops, ntop, id, s);
        }
        if (!split) {
            if (buf) for (int i = s + lane; i < e; i += 32) move_point(A, i, P0, i);
            __syncwarp();
            continue;
        }
        // Stable partition into the other buffer.
        int lbase = s, rbase = mid;
        const unsigned lt = (1u << lane) - 1u;
        for (int base = s; base < e; base += 32) {
            int i = base + lane;
            bool valid = i < e;
            bool left = false;
            if (valid) {
                // Rank of point i by (coordinate, position): the mid - s smallest go left.
                double c = axis == 2 ? A.z[i] : axis == 1 ? A.y[i] : A.x[i];
                int rank = 0;
                for (int j = s; j < e; ++j) {
                    double cj = axis == 2 ? A.z[j] : axis == 1 ? A.y[j] : A.x[j];
                    rank += (cj < c || (cj == c && j < i)) ? 1 : 0;
                }
                left = rank < (mid - s);
            }
            unsigned bl = __ballot_sync(0xffffffffu, valid && left);
            unsigned br = __ballot_sync(0xffffffffu, valid && !left);
            if (valid) {
                int dst = left ? lbase + __popc(bl & lt) : rbase + __popc(br & lt);
                if (dst < e) move_point(A, i, B, dst);
            }
            lbase += __popc(bl);
            rbase += __popc(br);
        }
        __syncwarp();
        // Push right then left (left is processed first).
        if (lane == 0) {
            int nb = buf ^ 1;
            WTask R = {mid, e, id, pack_meta(1, intop, nb, mintop - 1, maxtop - 1)};
            WTask L = {s, mid, id, pack_meta(0, intop, nb, mintop - 1, maxtop - 1)};
            if (sp + 2 > root.e - root.s) set_err(err, DEV_TASK_OVERFLOW);
            else { stk[sp] = R; stk[sp + 1] = L; }
        }
        sp += 2;
        if (sp > root.e - root.s) break;
        __syncwarp();
    }
}

template <bool FLATC, bool CPLX>
static int subtree_launch(int ntask, const BuildTask* tasks, Points P0, Points P1,
                          const BuildParams& BP, const Cells& C, int* tops, int* ntop,
                          WTask* wstack, int thread_t, int* err, cudaStream_t st)
{
    TC_TRY((allow_smem(k_subtree<FLATC, CPLX>, sizeof(SubShared))));
    count_launch();
    k_subtree<FLATC, CPLX><<<ntask, SB, sizeof(SubShared), st>>>(tasks, P0, P1, BP, C, tops, ntop,
                                                                 wstack, thread_t, err);
    TC_CU(cudaGetLastError());
    return 0;
}

static int launch_subtrees(int ntask, const BuildTask* tasks, Points P0, Points P1,
                           const BuildParams& BP, const Cells& C, int* tops, int* ntop,
                           WTask* wstack, int thread_t, int* err, cudaStream_t st)
{
    const bool flat = BP.coords == FLAT, cplx = BP.dkind == DG;
    auto* f = flat ? (cplx ? subtree_launch<true, true> : subtree_launch<true, false>)
                   : (cplx ? subtree_launch<false, true> : subtree_launch<false, false>);
    return f(ntask, tasks, P0, P1, BP, C, tops, ntop, wstack, thread_t, err, st);
}
// ---------------------------------------------------------------------------------------
// Structural check of the finished tree: every internal cell has two children that split
// its point range exactly.  This guarantees that the traversal (which only descends into
// children) terminates; the traversal is not launched on a tree that fails it.

__global__ void k_validate_tree(int ncap, Cells C, const int* tops, int ntop, int* err)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ntop) {
        int t = tops[i];
        if (t < 0 || t >= ncap) set_err(err, DEV_BAD_CHILD);
    }
    if (i >= ncap) return;
    int L = C.left[i], R = C.right[i];
    if (L < 0 && R < 0) return;
    if (L < 0 || R < 0 || L >= ncap || R >= ncap || L == i || R == i) {
        set_err(err, DEV_BAD_CHILD);
        return;
    }
    int n = C.n[i], nl = C.n[L], nr = C.n[R];
    if (nl < 1 || nr < 1 || nl + nr != n || C.start[L] != C.start[i] ||
        C.start[R] != C.start[i] + nl)
        set_err(err, DEV_BAD_CHILD);
}

void launch_validate_tree(int ncap, const Cells& C, const int* tops, int ntop, int* err,
                          cudaStream_t st)
{
    int m = ncap > ntop ? ncap : ntop;
    if (m <= 0) return;
    count_launch(); k_validate_tree<<<(m + 255) / 256, 256, 0, st>>>(ncap, C, tops, ntop, err);
}

// ---------------------------------------------------------------------------------------
// Host orchestration.

// Points per chunk and most points of a cell left to one block: the largest up to CH and SMALL,
// and for fewer than 300 SMALL points as much smaller as gives two blocks to every SM (FP64 runs at
// 2 lanes per clock and SM, so that the work has to be spread).
// Whole builds of a spin-2 field on the sphere, against chunks of 4096 and cells of 2048 points with
// the host in every level: 25,000 points 1.63 -> 0.93 ms, 200,000 2.0 -> 1.55, 10M 43.9 -> 40.5.
// Chunks from 256 points instead of 512: 25,000 points another 0.04 ms less.
constexpr int BUILD_LEVELS = 64;    // levels counted before the host looks again at the latest

static int spread(int n, int least, int most)
{
    const int want = n / 304;
    int v = least;
    while (v < want && v < most) v <<= 1;
    return std::min(v, most);
}

// Arrays for the cooperative levels of n points (a level's cells are disjoint, each above L.sub
// points).
static int scratch_levels(int n, BuildScratch& S, cudaStream_t st)
{
    if (S.level_mem) return 0;
    LevelBufs& L = S.L;
    L.ch = spread(n, 256, CH);
    L.sub = spread(n, 256, SMALL);
    L.cap_tasks = n / L.sub + 2;
    L.cap_chunks = n / L.ch + L.cap_tasks + 1;
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
    const size_t nt = L.cap_tasks, nc = L.cap_chunks;
    const size_t o_cnt = take(sizeof(int2) * (BUILD_LEVELS + 1)), o_small = take(sizeof(int)), o_done = take(sizeof(int) * nt);
    const size_t zeroed = off;
    const size_t o_t0 = take(sizeof(BuildTask) * nt), o_t1 = take(sizeof(BuildTask) * nt);
    const size_t o_k0 = take(sizeof(int2) * nt), o_k1 = take(sizeof(int2) * nt);
    const size_t o_c0 = take(sizeof(Chunk) * nc), o_c1 = take(sizeof(Chunk) * nc);
    const size_t o_p1 = take(sizeof(Part1) * nc), o_p2 = take(sizeof(Part2) * nc);
    const size_t o_st = take(sizeof(TaskStats) * nt);
    unsigned char* m = nullptr;
    TC_TRY(dalloc(&m, off));
    S.level_mem = m;
    L.cnt = reinterpret_cast<int2*>(m + o_cnt);
    L.nsmall = reinterpret_cast<int*>(m + o_small);
    L.done = reinterpret_cast<int*>(m + o_done);
    L.tasks[0] = reinterpret_cast<BuildTask*>(m + o_t0);
    L.tasks[1] = reinterpret_cast<BuildTask*>(m + o_t1);
    L.tchunk[0] = reinterpret_cast<int2*>(m + o_k0);
    L.tchunk[1] = reinterpret_cast<int2*>(m + o_k1);
    L.chunks[0] = reinterpret_cast<Chunk*>(m + o_c0);
    L.chunks[1] = reinterpret_cast<Chunk*>(m + o_c1);
    L.part1 = reinterpret_cast<Part1*>(m + o_p1);
    L.part2 = reinterpret_cast<Part2*>(m + o_p2);
    L.stats = reinterpret_cast<TaskStats*>(m + o_st);
    TC_CU(cudaMemsetAsync(m, 0, zeroed, st));
    return 0;
}

// *nc: the root's chunks.
static int launch_root(const BuildTask& root, const LevelBufs& L, int* nc, cudaStream_t st)
{
    *nc = (root.e - root.s + L.ch - 1) / L.ch;
    count_launch();
    k_level_root<<<(*nc + 255) / 256, 256, 0, st>>>(L, root);
    TC_CU(cudaGetLastError());
    return 0;
}

// 27 small kernels follow each other in a build of 25,000 points, 2 us apart: launch_chained takes
// whole builds of spin-2 points on the sphere from 0.67 to 0.60 ms there, 5000 from 0.59 to 0.52, 200,000
// from 1.40 to 1.32 and 10^6 from 4.51 to 4.46.
// The levels that even splits need, and a few more, go into the queue before the host looks;
// the kernels of levels without tasks return at once.
static int queue_levels(const TreeBuild& B, BuildRun& R, cudaStream_t st)
{
    const LevelBufs& L = B.S->L;
    const int n = B.BP.n;
    for (const int end = std::min(R.lev + R.batch, BUILD_LEVELS); R.lev < end; ++R.lev, ++R.total) {
        // No more than 2^level tasks: most chunks of a level, so the grid.
        const int tasks = R.total < 30 ? std::min(1 << R.total, L.cap_tasks) : L.cap_tasks;
        const int nc = std::min(n / L.ch + tasks, L.cap_chunks);
        TC_TRY(launch_chained(k_chunk_pass1, nc, CB, 0, st, L, R.lev, B.bufs[0], B.bufs[1], B.BP));
        TC_TRY(launch_chained(k_chunk_pass2, nc, CB, 0, st, L, R.lev, B.bufs[0], B.bufs[1], B.BP, B.C,
                              B.d_tops, B.d_ntop, B.d_err, 0));
        TC_TRY(launch_chained(k_chunk_scatter, nc, CB, 0, st, L, R.lev, B.bufs[0], B.bufs[1]));
    }
    R.batch = 8;
    TC_CU(cudaGetLastError());
    return 0;
}

int tree_begin(const TreeBuild& B, BuildRun& R, BuildRead* to, cudaMemcpyKind kind, cudaStream_t st)
{
    const int n = B.BP.n;
    BuildTask root;
    root.s = 0; root.e = n; root.parent = -1; root.side = 0;
    root.mintop = B.mintop; root.maxtop = B.maxtop; root.intop = 1; root.buf = 0;
    TC_TRY(scratch_levels(n, *B.S, st));
    const LevelBufs& L = B.S->L;
    TC_CU(cudaMemsetAsync(B.d_ntop, 0, sizeof(int), st));
    TC_CU(cudaMemsetAsync(L.cnt, 0, sizeof(int2) * (BUILD_LEVELS + 1), st));   // (field_center's)
    TC_CU(cudaMemsetAsync(L.nsmall, 0, sizeof(int), st));
    if (n > SMALL && B.BP.split == MEDIAN) {
        count_launch();
        k_median_levels<<<1, 32, 0, st>>>(root, B.bufs[0], B.bufs[1], B.BP, B.C, B.d_tops, B.d_ntop,
                                          B.S->wstack, L.small, L.nsmall, B.d_err);
        TC_CU(cudaGetLastError());
    } else if (n <= L.sub || B.BP.split == MEDIAN) {
        TC_CU(cudaMemcpyAsync(L.small, &root, sizeof(BuildTask), cudaMemcpyHostToDevice, st));
        R.whole = true;
        return 0;
    } else {
        int nc = 0;
        TC_TRY(launch_root(root, L, &nc, st));
        R.batch = 2;
        for (int m = L.sub; m < n; m = m > (1 << 29) ? n : 2 * m) ++R.batch;
        TC_TRY(queue_levels(B, R, st));
    }
    TC_CU(cudaMemcpyAsync(&to->left, L.cnt + R.lev, sizeof(int2), kind, st));
    TC_CU(cudaMemcpyAsync(&to->nsmall, L.nsmall, sizeof(int), kind, st));
    return 0;
}

int tree_subtrees(const TreeBuild& B, BuildRun& R, const BuildRead& read, BuildRead* to,
                  cudaMemcpyKind kind, cudaStream_t st)
{
    const LevelBufs& L = B.S->L;
    const int n = B.BP.n;
    int2 left = read.left;
    int nsmall = read.nsmall;
    if (R.whole) { left = make_int2(0, 0); nsmall = 1; }
    while (left.x != 0) {
        if (R.lev == BUILD_LEVELS) {
            // (an even number of levels: the arrays' turns go on)
            TC_CU(cudaMemsetAsync(L.cnt, 0, sizeof(int2) * (BUILD_LEVELS + 1), st));
            TC_CU(cudaMemcpyAsync(L.cnt, &left, sizeof(int2), cudaMemcpyHostToDevice, st));
            TC_CU(cudaStreamSynchronize(st));
            R.lev = 0;
        }
        TC_TRY(queue_levels(B, R, st));
        TC_CU(cudaMemcpyAsync(&left, L.cnt + R.lev, sizeof(int2), cudaMemcpyDeviceToHost, st));
        TC_CU(cudaMemcpyAsync(&nsmall, L.nsmall, sizeof(int), cudaMemcpyDeviceToHost, st));
        TC_CU(cudaStreamSynchronize(st));
    }
    if (nsmall > 0)
        TC_TRY(launch_subtrees(nsmall, L.small, B.bufs[0], B.bufs[1], B.BP, B.C, B.d_tops, B.d_ntop,
                               B.S->wstack, L.sub <= FEW_SUB ? THREAD_FEW : THREAD_T, B.d_err, st));
    launch_pack_cells(2 * n - 1, B.C, B.tcells, st);
    TC_CU(cudaGetLastError());
    TC_CU(cudaMemcpyAsync(&to->ntop, B.d_ntop, sizeof(int), kind, st));
    TC_CU(cudaMemcpyAsync(to->tops, B.d_tops, sizeof(int2) * std::min(n, BuildRead::FIRST), kind, st));
    return 0;
}

int tree_tops(const TreeBuild& B, const BuildRead& read, cudaStream_t st, std::vector<int>& tops_out)
{
    const int ntop = read.ntop;
    std::vector<std::pair<int, int>> v(ntop);
    std::vector<int2> more;
    if (ntop > BuildRead::FIRST) {
        more.resize(ntop);
        TC_CU(cudaMemcpyAsync(more.data(), B.d_tops, sizeof(int2) * ntop, cudaMemcpyDeviceToHost, st));
        TC_CU(cudaStreamSynchronize(st));
    }
    const int2* pairs = ntop > BuildRead::FIRST ? more.data() : read.tops;
    // Tops in the reference's depth-first order = increasing first point (left before right).
    for (int k = 0; k < ntop; ++k) v[k] = {pairs[k].x, pairs[k].y};
    std::sort(v.begin(), v.end());
    tops_out.resize(ntop);
    for (int k = 0; k < ntop; ++k) tops_out[k] = v[k].second;
    return 0;
}

void launch_prepare(int n, int coords, int dkind, const double* x, const double* y,
                    const double* z, const double* d1, const double* d2, const double* w,
                    const double* wpos, Points P, cudaStream_t st)
{
    if (n <= 0) return;
    count_launch(); k_prepare<<<(n + 255) / 256, 256, 0, st>>>(n, coords, dkind, x, y, z, d1, d2, w, wpos, P);
}

// Overall centre and size of the catalog (Field::Field, src/Field.cpp:198-203):
// one deterministic cooperative task over [0,n).
int field_center(const BuildParams& BP, Points P, BuildScratch& S, cudaStream_t st,
                 double out[4])
{
    const int n = BP.n;
    BuildTask root;
    root.s = 0; root.e = n; root.parent = -1; root.side = 0;
    root.mintop = 0; root.maxtop = 0; root.intop = 0; root.buf = 0;
    TC_TRY(scratch_levels(n, S, st));
    BuildParams B2 = BP;
    B2.split = MEAN;
    int nc = 0;
    TC_TRY(launch_root(root, S.L, &nc, st));
    TC_TRY(launch_chained(k_chunk_pass1, nc, CB, 0, st, S.L, 0, P, P, B2));
    TC_TRY(launch_chained(k_chunk_pass2, nc, CB, 0, st, S.L, 0, P, P, B2, Cells{}, nullptr, nullptr,
                          nullptr, 1));
    TC_CU(cudaGetLastError());
    TaskStats ts;
    TC_CU(cudaMemcpyAsync(&ts, S.L.stats, sizeof(TaskStats), cudaMemcpyDeviceToHost, st));
    TC_CU(cudaStreamSynchronize(st));
    out[0] = ts.cx; out[1] = ts.cy; out[2] = ts.cz; out[3] = ts.sizesq;
    return 0;
}

}  // namespace tc
