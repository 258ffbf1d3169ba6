// tile_packed.cu -- leaf-pair tiles of the exact mode for the common classes (NN; NK and KK; GG
// on flat and spherical coordinates): the pairs of k_tiles (tiles.cu), two per lane and step.
//
// One warp per tile.  A lane keeps one leaf of cell A in registers and walks B's leaves, two
// at a time, as packed FP32 pairs (fma.rn.f32x2 and its kin): one instruction for two pairs,
// and B's leaves, the same for all lanes, come as broadcast loads of shared memory.  k_tiles
// gives every lane another pair of leaves instead and reads both from shared memory.
// When A has more than 32 leaves, the rest share the lanes: 32 / r lanes to each of r leaves,
// B's pairs dealt out among them.
//
// The tile's bounds (k_tile_class) decide how its pairs are binned.  All in one bin: sums in
// registers.  All in two bins: one comparison, sums in registers.  Anything else (more bins, the
// ends of the range, the diagonal, leaves of several points): every lane adds into its own
// column of a histogram in shared memory, 6 (GG), 12 or 16 bins wide, moved along when the tile
// reaches further; a column is one bank set, so the additions need no atomics, do not
// conflict and have a fixed order.  Only a pair within the FP32 error of a bin edge leaves the
// loop: it goes onto a list and is decided after it in FP64 from the FP64 positions
// (leaf_pair64), like every pair of a tile whose list overflows.  Same bounds and bands as
// k_tiles.
//
// Measured against k_tiles, tile kernels of GG on the full sphere, 30 bins, 1' to 300', bin_slop
// 0: 10^6 points 278.7 -> 148.3 ms, 200,000 points 27.5 -> 9.0 ms; with 10 bins 189.2 -> 119.3 and
// 14.9 -> 7.0 ms, with 100 bins 1308 -> 300 and 86.2 -> 25.3 ms; NN of 10^6 points 233.7 -> 96.1,
// KK of 200,000 25.5 -> 5.8 ms.  In the histogram form a step of 64 pairs takes 48 packed FP32
// instructions (two FMA-pipe cycles each), 8 reciprocals, roots and logarithms and 32 + 6
// shared-memory cycles per warp, so FMA pipe (49% busy), shared memory (67%) and issue slots
// (59%) are near balance; the rest is latency at the 16 warps that registers and shared memory
// leave room for, and one lane in six idle where cells hold fewer than 32 leaves.
// Not kept: four register bins at a time for the wide tiles (204 ms), three register bins as
// well as the histogram (165 ms against 158), a kernel per class (222 ms: staging is repeated and
// each grid has its own tail), all in one kernel with unrolled forms of 4-6 KB each (277 ms: a
// third of the time waiting for instructions).
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "tc_internal.cuh"
#include "tc_host.hpp"
#include "traverse2pt.hpp"
#include "pair_math.cuh"
#include "tile_common.cuh"

namespace tc {

namespace {

constexpr int PB = 128;             // threads per block
constexpr int PW = PB / 32;
constexpr int PMINB = 4;            // resident blocks the registers and shared memory are sized for:
                                    // 3 (8 rows per histogram) 162 ms, 5 (4 rows) 168 ms
constexpr int PFLUSH = 8;           // tiles between flushes of the FP32 bins
constexpr int PLEAF = 64;           // most leaves per side (>= the traversal's tile_leaf)
constexpr int PPAIRS = 40;          // pairs of B leaves: 32, and up to 8 empty ones that round
                                    // their number up to a multiple of the lane groups
constexpr int PESC = 64;            // listed pairs per tile

// Two FP32 values in one 64-bit register.
typedef unsigned long long f2;
__device__ __forceinline__ f2 mk2(float a, float b)
{ f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ f2 mk2(float a) { return mk2(a, a); }
__device__ __forceinline__ float lo2(f2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(f2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{ f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{ f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{ f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

// The approximations without their detours for subnormal arguments (packed_tiles admits only
// traversals whose squared separations are normal).
__device__ __forceinline__ f2 rsqrt2(f2 a)
{
    float x, y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(lo2(a)));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(hi2(a)));
    return mk2(x, y);
}
__device__ __forceinline__ f2 rcp2(f2 a)
{
    float x, y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(lo2(a)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(hi2(a)));
    return mk2(x, y);
}
__device__ __forceinline__ f2 log2_2(f2 a)
{
    float x, y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(lo2(a)));
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(hi2(a)));
    return mk2(x, y);
}

// Two leaves of B: minus the offset from B's centre, half the z coordinate, weight, payload.
struct __align__(16) BPair {
    f2 nx, ny;
    f2 nz, zh;
    f2 w, p1;
    f2 p2, np2;      // and minus the imaginary part
};
struct BSlot { BPair v; int4 gap; };    // 80 bytes apart: staging stores meet in a bank two at a
                                        // time (64 bytes apart: eight)
static_assert(sizeof(BSlot) == 80, "");

struct PackedSide {
    BSlot b[PPAIRS];
    int nbl[2 * PPAIRS];                    // point count (0: empty)
    unsigned short esc[PESC];               // i << 8 | j
    unsigned char ib[2 * PPAIRS], ia[PLEAF];    // the leaves' places in their cells
};
static_assert(sizeof(PackedSide) % 16 == 0, "");

struct PTile {
    int na, nj, kref, idA, idB;             // id*: leaf cell ids of the cells' first points
    float inv_edge, emax, band_e, band_0, chx, chy, chz, clx, cly, clz;
    bool self, special;
};

// Listed pairs (or, all = true, every pair of the tile), decided and added in FP64 / FP32 as
// the reference does, into the warp's shared-memory bins in ascending order.
// Returns how many this lane accepted and decided.
__device__ __noinline__ uint2 packed_slow(const TravParams& T, const PackedSide& S, int idA,
                                          int idB, int na, int nbl, bool self, bool all,
                                          int count, float* fb,
                                          unsigned long long* np, int lane)
{
    unsigned acc = 0, esc = 0;
    const int total = all ? na * nbl : count;
    for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int kx = -1;
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const int e = t < total && !all ? S.esc[t] : 0;
        const int i = all ? t / nbl : e >> 8, j = all ? t - (t / nbl) * nbl : e & 0xff;
        if (t < total && !(self && j <= i)) {
            const int ida = idA + S.ia[i], idb = idB + S.ib[j];
            float r = 0.f, logr = 0.f;
            ++esc;
            kx = leaf_pair64(T, ida, idb, self, &r, &logr);
            if (kx >= 0) {
                const TCell A = T.c1[ida], B = (self ? T.c1 : T.c2)[idb];
                const float dx = (A.a.x - B.a.x) + (A.b.x - B.b.x);
                const float dy = (A.a.y - B.a.y) + (A.b.y - B.b.y);
                const float dz = T.coords == FLAT ? 0.f : (A.a.z - B.a.z) + (A.b.z - B.b.z);
                float av[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                unsigned long long nn = 0;
                accept_values(T, A, B, ida, idb, dx, dy, dz, dx * dx + dy * dy + dz * dz, r, logr,
                              av, nn);
#pragma unroll
                for (int q = 0; q < 7; ++q) v[q] = av[q];
                ++acc;
                if (!T.quick) atomicAdd(&np[kx], nn);
            }
        }
        shared_bins_in_order(kx, v, fb, T.nqf, T.nbins, lane);
        __syncwarp();
    }
    return make_uint2(acc, esc);
}

// Lists the pairs (i, j) where u0 is set and (i, j + 1) where u1 is.
__device__ __forceinline__ void list_pairs(PackedSide& S, bool u0, bool u1, int i, int j,
                                           int& ecount, int lane)
{
    const unsigned m0 = __ballot_sync(0xffffffffu, u0), m1 = __ballot_sync(0xffffffffu, u1);
    const unsigned lt = (1u << lane) - 1u;
    const int o0 = ecount + __popc(m0 & lt), o1 = ecount + __popc(m0) + __popc(m1 & lt);
    if (u0 && o0 < PESC) S.esc[o0] = (unsigned short)((i << 8) | j);
    if (u1 && o1 < PESC) S.esc[o1] = (unsigned short)((i << 8) | (j + 1));
    ecount += __popc(m0) + __popc(m1);
}

// A lane's leaf of A: its offset from B's centre, weight and payload (0 for an idle lane).
struct PRow {
    f2 ax, ay, az, aw, ar, ai, nai, X, nY, nazh;
    int i, grp;
    bool on;
    unsigned n;
};

__device__ __forceinline__ void load_row(const TravParams& T, const PackedSide& S, const PTile& C,
                                         int i0, int groups, int rows, int lane, PRow& A)
{
    A.grp = (int)((lane + 0.5f) * __frcp_rn((float)rows));
    A.on = A.grp < groups;
    A.i = A.on ? i0 + lane - A.grp * rows : i0;
    if (!A.on) A.grp = 0;
    const int id = C.idA + S.ia[A.i];
    const float4 a = T.c1[id].a, b = T.c1[id].b, c = T.c1[id].c;
    A.n = A.on ? (unsigned)__float_as_int(c.z) : 0u;
    const float p1 = T.k1 == DN ? b.w : c.x;
    A.ax = mk2((a.x - C.chx) + (b.x - C.clx));
    A.ay = mk2((a.y - C.chy) + (b.y - C.cly));
    A.az = mk2((a.z - C.chz) + (b.z - C.clz));
    A.aw = mk2(A.on ? b.w : 0.f);
    A.ar = mk2(A.on ? p1 : 0.f);
    A.ai = mk2(A.on ? c.y : 0.f);
    A.nai = mk2(A.on ? -c.y : 0.f);
    A.X = mk2(a.x);
    A.nY = mk2(-a.y);
    A.nazh = mk2(-0.5f * a.z);
}

template <int KIND>
__device__ __forceinline__ BPair load_pair(const PackedSide& S, int jp)
{
    BPair B;
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(&S.b[jp].v);
    const ulonglong2 v0 = p[0], v1 = p[1], v2 = p[2];
    B.nx = v0.x; B.ny = v0.y; B.nz = v1.x; B.zh = v1.y; B.w = v2.x; B.p1 = v2.y;
    B.p2 = B.np2 = 0ull;
    if (KIND == TK_GG) { const ulonglong2 v3 = p[3]; B.p2 = v3.x; B.np2 = v3.y; }
    return B;
}

// Two pairs' separations r, log2(r^2 / edge^2) lr, reciprocal chord ic, weight ww and products:
// x, or for GG on the sphere their factors (products<>()).
struct PVals { f2 r, lr, ic, ww, x[4]; };

// SPECIAL: chords of 0.25 and more, or a pole in reach (k_tile_class).
template <int GEO, int KIND, bool SPECIAL>
__device__ __forceinline__ void pair_vals(const PTile& C, const PRow& A, const BPair& B, PVals& V)
{
    const f2 one = mk2(1.f), mone = mk2(-1.f);
    const f2 dx = add2(A.ax, B.nx), dy = add2(A.ay, B.ny);
    f2 dsq, dz = 0ull;
    if (GEO == TG_FLAT) {
        dsq = fma2(dx, dx, mul2(dy, dy));
    } else {
        dz = add2(A.az, B.nz);
        dsq = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    }
    V.ic = rsqrt2(dsq);
    f2 r = mul2(dsq, V.ic);
    if (GEO == TG_ARC) {
        // 2 asin(c / 2) by its series in c^2 (arc_series)
        f2 p = fma2(dsq, mk2(5.f / 7168.f), mk2(3.f / 640.f));
        p = fma2(dsq, p, mk2(1.f / 24.f));
        r = mul2(r, fma2(dsq, p, one));
        if (SPECIAL) r = mk2(arc_from_chord_sq(lo2(dsq)), arc_from_chord_sq(hi2(dsq)));
    }
    V.r = r;
    V.lr = log2_2(mul2(GEO == TG_ARC ? mul2(r, r) : dsq, mk2(C.inv_edge)));
    V.ww = mul2(A.aw, B.w);
    if constexpr (KIND == TK_SC) {
        V.x[0] = mul2(A.ar, B.p1);                              // wk1 wk2
    } else if constexpr (KIND == TK_GG && GEO == TG_FLAT) {
        // as pair_products: g1 conj(g2), and g1 g2 turned by conj(r)^4 / |r|^4
        V.x[0] = fma2(A.ar, B.p1, mul2(A.ai, B.p2));
        V.x[1] = fma2(A.ai, B.p1, mul2(A.ar, B.np2));
        const f2 q = rcp2(dsq);
        const f2 er = mul2(fma2(dx, dx, mul2(mul2(dy, dy), mone)), q);
        const f2 ei = mul2(mul2(dx, dy), mul2(q, mk2(-2.f)));
        const f2 e2r = fma2(er, er, mul2(mul2(ei, ei), mone)), e2i = mul2(mul2(er, ei), mk2(2.f));
        const f2 pr = fma2(A.ar, B.p1, mul2(A.ai, B.np2)), pi = fma2(A.ar, B.p2, mul2(A.ai, B.p1));
        V.x[2] = fma2(pr, e2r, mul2(mul2(pi, e2i), mone));
        V.x[3] = fma2(pr, e2i, mul2(pi, e2r));
    } else if constexpr (KIND == TK_GG) {
        // as pair_products, with both phases negated (their product is unchanged):
        // E = (cos^2 - sin^2, -2 sin cos) at either end, cosB with its sign changed.
        const f2 sinA = fma2(A.X, dy, mul2(A.nY, dx));
        const f2 cosA = fma2(B.zh, dsq, dz);
        const f2 cosB = fma2(A.nazh, dsq, dz);
        const f2 s2 = mul2(sinA, sinA), tS = mul2(sinA, mk2(-2.f));
        f2 m2 = fma2(cosA, cosA, s2), m1 = fma2(cosB, cosB, s2);
        if (SPECIAL) { m2 = add2(m2, mk2(POLE_SQ)); m1 = add2(m1, mk2(POLE_SQ)); }
        const f2 E2r = fma2(s2, mk2(-2.f), m2), E2i = mul2(tS, cosA);
        const f2 E1r = fma2(s2, mk2(-2.f), m1), E1i = mul2(tS, cosB);
        const f2 i2 = rcp2(m2), i1 = rcp2(m1);
        V.x[0] = mul2(fma2(B.p1, E2r, mul2(B.np2, E2i)), i2);
        V.x[1] = mul2(fma2(B.p1, E2i, mul2(B.p2, E2r)), i2);
        V.x[2] = mul2(fma2(A.ar, E1r, mul2(A.nai, E1i)), i1);
        V.x[3] = mul2(fma2(A.ar, E1i, mul2(A.ai, E1r)), i1);
    }
}

// Sphere GG: of g2 = x0 + i x1 and g1 = x2 + i x3 the four real products are summed, and made
// into xi+ and xi- (accept_values) by sphere_gg() at the end of the tile.
template <int GEO, int KIND>
__device__ __forceinline__ f2 product(const PVals& V, int q)
{
    if constexpr (KIND == TK_GG && GEO != TG_FLAT)
        return mul2(V.x[q == 0 || q == 2 ? 0 : 1], V.x[q == 0 || q == 3 ? 2 : 3]);
    return V.x[q];
}

template <int GEO, int KIND>
__device__ __forceinline__ f2 add_product(const PVals& V, int q, f2 acc)
{
    if constexpr (KIND == TK_GG && GEO != TG_FLAT)
        return fma2(V.x[q == 0 || q == 2 ? 0 : 1], V.x[q == 0 || q == 3 ? 2 : 3], acc);
    return add2(acc, V.x[q]);
}

template <int GEO, int KIND>
__device__ __forceinline__ void sphere_gg(float (&o)[8])
{
    if constexpr (KIND == TK_GG && GEO != TG_FLAT) {
        // o[3..6]: re re, im im, re im (g2 g1), im re
        const float rr = o[3], ii = o[4], ri = o[5], ir = o[6];
        o[3] = rr + ii; o[4] = ri - ir; o[5] = rr - ii; o[6] = ri + ir;
    }
}

// All pairs of a tile whose pairs lie in range and in bins kref .. kref + NB - 1 (NB = 2: and
// whose leaves hold one point each).  Returns the lane's sums per bin, and its count of pairs of
// bin kref + 1 in cn.  Pairs within the error of a bin edge are listed and left out.
template <int GEO, int KIND, int NB>
__device__ __forceinline__ void packed_pairs(const TravParams& T, PackedSide& S, const PTile& C,
                                             int lane, float (&out)[NB][8], unsigned& cn,
                                             int& ecount)
{
    constexpr int NX = KIND == TK_NN ? 0 : KIND == TK_SC ? 1 : 4;
    constexpr int NV = 3 + NX;
    f2 acc2[NB][NV];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
        for (int q = 0; q < NV; ++q) acc2[b][q] = 0ull;
    }
    cn = 0u;
    const float ckk = 0.5f * 0.69314718f * T.finvbinsize;   // bins per unit of log2(r^2)
    const f2 one = mk2(1.f), mone = mk2(-1.f);
    const f2 band_e = mk2(C.band_e), band_0 = mk2(C.band_0);
    const int njp = (C.nj + 1) >> 1;
    for (int i0 = 0; i0 < C.na; i0 += 32) {
        // This round's leaves of A: lane -> (leaf, group).
        const int rows = min(32, C.na - i0);
        const int groups = 32 / rows;
        PRow A;
        load_row(T, S, C, i0, groups, rows, lane, A);
        f2 cf = 0ull;                           // pairs of bin kref + 1
        for (int t0 = 0; t0 < njp; t0 += groups) {
            const int jp = t0 + A.grp;
            const BPair B = load_pair<KIND>(S, jp);
            PVals V;
            pair_vals<GEO, KIND, false>(C, A, B, V);
            if constexpr (NB == 1) {
                acc2[0][0] = add2(acc2[0][0], V.ww);
                acc2[0][1] = fma2(V.ww, V.r, acc2[0][1]);
                acc2[0][2] = fma2(V.ww, V.lr, acc2[0][2]);
#pragma unroll
                for (int q = 0; q < NX; ++q) acc2[0][3 + q] = add_product<GEO, KIND>(V, q, acc2[0][3 + q]);
            } else {
                const f2 k = mul2(V.lr, mk2(ckk)), band = fma2(band_e, V.ic, band_0);
                const int2 n2 = *reinterpret_cast<const int2*>(&S.nbl[2 * jp]);
                const f2 leaf = mk2(n2.x ? 1.f : 0.f, n2.y ? 1.f : 0.f);
                const float k0 = lo2(k), k1 = hi2(k);
                bool u0 = fabsf(k0 - 1.f) < lo2(band), u1 = fabsf(k1 - 1.f) < hi2(band);
                f2 sure = one;
                if (__any_sync(0xffffffffu, u0 || u1)) {
                    if (u0 || u1) sure = mk2(u0 ? 0.f : 1.f, u1 ? 0.f : 1.f);
                    u0 = u0 && A.on && lo2(leaf) != 0.f;
                    u1 = u1 && A.on && hi2(leaf) != 0.f;
                    list_pairs(S, u0, u1, A.i, 2 * jp, ecount, lane);
                }
                const f2 up = mk2(k0 >= 1.f ? lo2(sure) : 0.f, k1 >= 1.f ? hi2(sure) : 0.f);
                const f2 m[2] = {fma2(up, mone, sure), up};
                cf = fma2(up, leaf, cf);
                f2 v[NV];
                v[0] = V.ww; v[1] = mul2(V.ww, V.r); v[2] = mul2(V.ww, V.lr);
#pragma unroll
                for (int q = 0; q < NX; ++q) v[3 + q] = product<GEO, KIND>(V, q);
#pragma unroll
                for (int b = 0; b < NB; ++b)
#pragma unroll
                    for (int q = 0; q < NV; ++q) acc2[b][q] = fma2(m[b], v[q], acc2[b][q]);
            }
        }
        if (NB > 1 && A.on) cn += (unsigned)(lo2(cf) + hi2(cf));
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            out[b][q] = q < NV ? lo2(acc2[b][q < NV ? q : 0]) + hi2(acc2[b][q < NV ? q : 0]) : 0.f;
        sphere_gg<GEO, KIND>(out[b]);
    }
}

// The general form: each lane adds its pairs into a column of its own of a histogram in shared
// memory, rows for bins kref + w0 .. + hist_rows - 1 and one for what is left out.  A row of a
// column: weight, w r, w lr, point pairs (an integer); the products (1, or 4).  Pairs out of
// range have no row or, near its ends, are listed: the ends are bin edges (packed_tiles).
template <int KIND> __host__ __device__ constexpr int hist_rows()
{ return KIND == TK_NN ? 16 : KIND == TK_SC ? 12 : 6; }
template <int KIND> __host__ __device__ constexpr int hist_words()
{ return KIND == TK_NN ? 4 : KIND == TK_SC ? 5 : 8; }
template <int KIND> __host__ __device__ constexpr size_t hist_bytes()
{ return sizeof(float) * 32 * hist_words<KIND>() * (hist_rows<KIND>() + 1); }

template <int GEO, int KIND, bool SPECIAL>
__device__ __forceinline__ void packed_hist(const TravParams& T, PackedSide& S, const PTile& C,
                                            float* hist, int lane, int w0, int& ecount,
                                            unsigned& n_acc)
{
    constexpr int NX = KIND == TK_NN ? 0 : KIND == TK_SC ? 1 : 4;
    constexpr int W = hist_rows<KIND>(), RF = 32 * hist_words<KIND>();   // floats per row
    const f2 ckk = mk2(0.5f * 0.69314718f * T.finvbinsize), half = mk2(-0.5f);
    const f2 big = mk2(12582912.f), nbig = mk2(-12582912.f), mone = mk2(-1.f);
    const f2 nband_e = mk2(-C.band_e), hband = mk2(0.5f - C.band_0);
    const unsigned wlim = (unsigned)min(W, T.nbins - C.kref - w0);
    const int njp = (C.nj + 1) >> 1;
    unsigned char* h0 = reinterpret_cast<unsigned char*>(hist) + 16 * lane;
    unsigned char* h1 = reinterpret_cast<unsigned char*>(hist) + 512 + (NX == 4 ? 16 : 4) * lane;
    for (int i0 = 0; i0 < C.na; i0 += 32) {
        const int rows = min(32, C.na - i0);
        const int groups = 32 / rows;
        PRow A;
        load_row(T, S, C, i0, groups, rows, lane, A);
        // This lane's pairs (i, j): j = js + 1 .. js + jn.
        const int js = C.self ? A.i : -1;
        const unsigned jn = A.on ? (unsigned)(C.nj - 1 - js) : 0u;
        for (int t0 = 0; t0 < njp; t0 += groups) {
            const int jp = t0 + A.grp;
            const BPair B = load_pair<KIND>(S, jp);
            PVals V;
            pair_vals<GEO, KIND, SPECIAL>(C, A, B, V);
            const uint2 n2 = *reinterpret_cast<const uint2*>(&S.nbl[2 * jp]);
            // floor(k) (adding 1.5 2^23 rounds to an integer); the distance to the nearer bin
            // edge is 0.5 - |g|.
            const f2 t = fma2(V.lr, ckk, half), m = add2(t, big), g = fma2(add2(m, nbig), mone, t);
            const f2 lim = fma2(nband_e, V.ic, hband);
            const unsigned j0 = 2 * jp - js - 1;
            const bool in0 = j0 < jn, in1 = j0 + 1u < jn;
            const bool s0 = fabsf(lo2(g)) <= lo2(lim), s1 = fabsf(hi2(g)) <= hi2(lim);
            const bool u0 = in0 && !s0, u1 = in1 && !s1;
            if (__any_sync(0xffffffffu, u0 || u1) && w0 == 0)
                list_pairs(S, u0, u1, A.i, 2 * jp, ecount, lane);
            const f2 wr = mul2(V.ww, V.r), wl = mul2(V.ww, V.lr);
            f2 x[NX > 0 ? NX : 1];
#pragma unroll
            for (int q = 0; q < NX; ++q) x[q] = product<GEO, KIND>(V, q);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // (what is left out may not be finite)
                const unsigned row = __float_as_uint(h ? hi2(m) : lo2(m)) - 0x4B400000u - (unsigned)w0;
                const bool ok = (h ? in1 && s1 : in0 && s0) && row < wlim;
                const unsigned at = (ok ? row : (unsigned)W) * (RF * 4);
                const unsigned nn = A.n * (h ? n2.y : n2.x);
                float4 a = *reinterpret_cast<const float4*>(h0 + at);
                a.x += h ? hi2(V.ww) : lo2(V.ww);
                a.y += h ? hi2(wr) : lo2(wr);
                a.z += h ? hi2(wl) : lo2(wl);
                a.w = __uint_as_float(__float_as_uint(a.w) + nn);
                if constexpr (NX == 4) {
                    float4 b = *reinterpret_cast<const float4*>(h1 + at);
                    b.x += h ? hi2(x[0]) : lo2(x[0]);
                    b.y += h ? hi2(x[1]) : lo2(x[1]);
                    b.z += h ? hi2(x[2]) : lo2(x[2]);
                    b.w += h ? hi2(x[3]) : lo2(x[3]);
                    *reinterpret_cast<float4*>(h1 + at) = b;
                } else if constexpr (NX == 1) {
                    *reinterpret_cast<float*>(h1 + at) += h ? hi2(x[0]) : lo2(x[0]);
                }
                *reinterpret_cast<float4*>(h0 + at) = a;
                n_acc += ok;
            }
        }
    }
}

template <int KIND> __host__ __device__ inline size_t packed_warp_bytes(int nq, int nb)
{ return bins_bytes(nq, nb) + sizeof(PackedSide) + hist_bytes<KIND>(); }

// What k_tile_class found for a tile, in 32 bits: the kernel that takes it (its NB, 0: no pair
// in range; 1, 2: bins; 3: the histogram), whether it is special (pair_vals), the lowest bin and
// how many bins above it the bounds reach.
__host__ __device__ inline unsigned tile_key(int cls, bool special, int klo, int span)
{ return (unsigned)cls | (special ? 16u : 0u) | ((unsigned)klo << 5) | ((unsigned)span << 18); }
constexpr int KEY_MAXNB = 8191;

// A drain of the tile list: the launch after the expansion that left no room for another
// chunk's tiles, or that ended the traversal (the launches in between return at once, so the
// list is worked off in few large launches).
__device__ __forceinline__ long long tiles_to_drain(const TravParams& T)
{
    long long nt = (long long)*(volatile unsigned long long*)&T.tctl[0];
    if (nt > T.tile_cap) nt = T.tile_cap;       // (the expansion raised DEV_SPILL_OVERFLOW)
    const bool done = *(volatile int*)&T.sched->done != 0;
    return done || nt > T.tile_drain ? nt : 0;
}

// The bounds of every waiting tile, one lane per tile.
template <int GEO>
__global__ void __launch_bounds__(256) k_tile_class(const __grid_constant__ TravParams T)
{
    const long long nt = tiles_to_drain(T);
    const int nb = T.nbins;
    const float ckk = 0.5f * 0.69314718f * T.finvbinsize;
    for (long long t = (long long)blockIdx.x * 256 + threadIdx.x; t < nt; t += (long long)gridDim.x * 256) {
        const int2 tile = T.tiles[t];
        const bool self = tile.y < 0;
        const TCell* cB = self ? T.c1 : T.c2;
        const int ia = tile.x, ib = self ? -2 - tile.y : tile.y;
        const float4 Aa = T.c1[ia].a, Ab = T.c1[ia].b, Ba = cB[ib].a, Bb = cB[ib].b;
        // Bounds of the tile's separations from the two cells' sizes (each point lies within
        // size of its cell's FP64 centre; 1e-6 covers the size's FP32 rounding), as in k_tiles.
        const float Dx = (Aa.x - Ba.x) + (Ab.x - Bb.x), Dy = (Aa.y - Ba.y) + (Ab.y - Bb.y);
        const float Dz = GEO == TG_FLAT ? 0.f : (Aa.z - Ba.z) + (Ab.z - Bb.z);
        const float Dsq = Dx * Dx + Dy * Dy + Dz * Dz;
        const float Dn = Dsq > 0.f ? Dsq * rsqrtf(Dsq) : 0.f;
        const float rAB = (Aa.w + Ba.w) * (1.f + 1e-6f) + 1e-30f;
        // emax bounds |FP32 d - d| of every pair: each offset within 2 ulps of its L1 size, the
        // difference one more (a 1.5x margin), and L1 <= sqrt(3) L2.
        const float emax = 4.7e-7f * (Dn + rAB) + 1e-30f;
        const float slack = emax + 2e-6f * (Dn + rAB);
        float lo = fmaxf(Dn - rAB - slack, 0.f), hi = Dn + rAB + slack;
        const bool small = hi < 0.25f;
        // Special tiles: chords of 0.25 and more (Arc), or for GG a direction that FP32 can cancel
        // to nothing.  That is |p1 - p2| cos(dec) sin(..), and its FP32 error some 2e-7 of
        // |p1 - p2| (cos(dec) + |p1 - p2|) at most: it is well above the error where every point is 1e-4
        // from the poles' axis and no pair near antipodal, and its square a normal number
        // from a min_sep of 1e-13 on (pick).
        const bool gg = (GEO == TG_ARC || GEO == TG_SPHEUC) && T.k2 == DG;
        const bool pole = gg && (sqrtf(Aa.x * Aa.x + Aa.y * Aa.y) - Aa.w <= 1e-4f ||
                                 sqrtf(Ba.x * Ba.x + Ba.y * Ba.y) - Ba.w <= 1e-4f || hi > 1.999f);
        const bool special = pole || (GEO == TG_ARC && !small);
        if (GEO == TG_ARC) {
            if (small) { lo = arc_series(lo); hi = arc_series(hi); }
            else { lo = arc_from_chord_sq(lo * lo); hi = arc_from_chord_sq(hi * hi); }
        }
        lo *= 1.f - 1e-5f;
        hi *= 1.f + 1e-5f;
        unsigned key = 0;
        float band_0 = 0.f;
        if (!(lo >= T.fmaxsep || hi < T.fminsep)) {
            const bool interior = lo >= T.fminsep && hi < T.fmaxsep;
            const float lb = fmaxf(lo, T.fminsep), hb = fminf(hi, T.fmaxsep);
            int klo = (int)floorf(__log2f(lb * lb * T.finvminsepsq) * ckk);
            int khi = (int)floorf(__log2f(hb * hb * T.finvminsepsq) * ckk);
            klo = klo < 0 ? 0 : (klo > nb - 1 ? nb - 1 : klo);
            khi = khi < 0 ? 0 : (khi > nb - 1 ? nb - 1 : khi);
            // Band (in bins) outside which the FP32 bin is certain: r's relative error
            // (emax / chord + 4e-7) and __log2f's (2^-22 absolute on [0.5, 2], else 2 ulps;
            // |log2| <= lmax here), the roundings of its argument and of kk.
            const float lmax = fmaxf(fabsf(__log2f(hi * hi * T.tile_edge[klo])), 1.f);
            band_0 = 4e-7f * T.finvbinsize + (5e-7f + 4.2e-7f * lmax) * ckk + 2e-7f;
            const bool plain = interior && !self && !special;
            const int span = khi - klo;
            key = tile_key(plain && span < 2 ? span + 1 : 3, special, klo, span);
        }
        T.tile_keys[t] = key;
        T.tile_err[t] = make_float2(emax, band_0);
    }
}

template <int GEO, int KIND>
__global__ void __launch_bounds__(PB, PMINB) k_tiles_packed(const __grid_constant__ TravParams T)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = blockIdx.x * PW + wib;
    const int nq = T.nqf, nb = T.nbins;
    const long long nt = tiles_to_drain(T);
    const long long nwt = (long long)gridDim.x * PW;
    unsigned char* wb = smem + (size_t)wib * packed_warp_bytes<KIND>(nq, nb);
    float2* fd = reinterpret_cast<float2*>(wb);
    unsigned long long* np = reinterpret_cast<unsigned long long*>(fd + nq * nb);
    float* fb = reinterpret_cast<float*>(np + nb);
    PackedSide& S = *reinterpret_cast<PackedSide*>(wb + bins_bytes(nq, nb));
    float* hist = reinterpret_cast<float*>(wb + bins_bytes(nq, nb) + sizeof(PackedSide));
    unsigned n_acc = 0, n_esc = 0, n_tiles = 0;
    unsigned long long n_sure = 0, n_pairs = 0;     // (uniform)
    // Warps take runs of tiles: 32, or fewer when there are not enough for all.
    const int run = (int)max(1ll, min(32ll, nt / nwt));
    const bool quick = T.quick != 0;
    int since_flush = -1;                            // -1: no tile yet
    for (long long g = (long long)gw * run; g < nt; g += nwt * run) {
        const unsigned my = lane < run && g + lane < nt ? T.tile_keys[g + lane] : 0u;
        unsigned todo = __ballot_sync(0xffffffffu, (my & 7u) != 0u);
        while (todo) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1u;
            const unsigned key = __shfl_sync(0xffffffffu, my, q);
            const int2 tile = T.tiles[g + q];
            const float2 err = T.tile_err[g + q];
            if (since_flush < 0) {
                for (int z = lane; z < nq * nb; z += 32) { fd[z] = make_float2(0.f, 0.f); fb[z] = 0.f; }
                for (int z = lane; z < nb; z += 32) np[z] = 0ull;
                __syncwarp();
                since_flush = 0;
            }
            PTile C;
            C.self = tile.y < 0;
            const int ia = tile.x, ib = C.self ? -2 - tile.y : tile.y;
            const TCell* cB = C.self ? T.c1 : T.c2;
            const int baseB = C.self ? T.leaf_base1 : T.leaf_base2;
            const int nA = __float_as_int(T.c1[ia].c.z), sA = __float_as_int(T.c1[ia].d.z);
            const float4 Ba = cB[ib].a, Bb = cB[ib].b;
            const int nB = __float_as_int(cB[ib].c.z), sB = __float_as_int(cB[ib].d.z);
            const int cls = key & 7u;
            C.special = (key & 16u) != 0u;
            C.kref = (key >> 5) & 8191u;
            const int span = (int)(key >> 18);
            C.inv_edge = T.tile_edge[C.kref];         // 1 / (lower edge of kref)^2
            const float ledge = T.tile_ledge[C.kref]; // log of that edge
            C.emax = err.x;
            C.band_e = err.x * T.finvbinsize;
            C.band_0 = err.y;
            C.chx = Ba.x; C.chy = Ba.y; C.chz = Ba.z;
            C.clx = Bb.x; C.cly = Bb.y; C.clz = Bb.z;
            C.idA = T.leaf_base1 + sA;
            C.idB = baseB + sB;
            // The leaves (n > 0, w != 0, in point order): ids of A's, all of B's.
            int na = 0, nj = 0;
            bool single = true;
            unsigned sumA = 0, sumB = 0;
            const unsigned lt = (1u << lane) - 1u;
#pragma unroll
            for (int h = 0; h < PLEAF / 32; ++h) {
                const int p = lane + 32 * h;
                if (32 * h >= nB) break;
                const int id = baseB + sB + p;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, c = a;
                if (p < nB) { a = cB[id].a; b = cB[id].b; c = cB[id].c; }
                const int n = __float_as_int(c.z);
                const bool v = n > 0 && b.w != 0.f;
                const unsigned m = __ballot_sync(0xffffffffu, v);
                single = single && __all_sync(0xffffffffu, !v || n == 1);
                if (v) {
                    const int o = nj + __popc(m & lt);
                    float* f = reinterpret_cast<float*>(&S.b[o >> 1]) + (o & 1);
                    f[0] = -((a.x - Ba.x) + (b.x - Bb.x));
                    f[2] = -((a.y - Ba.y) + (b.y - Bb.y));
                    f[4] = -((a.z - Ba.z) + (b.z - Bb.z));
                    f[6] = 0.5f * a.z;
                    f[8] = b.w;
                    f[10] = T.k2 == DN ? b.w : c.x;
                    f[12] = c.y;
                    f[14] = -c.y;
                    S.ib[o] = (unsigned char)p;
                    S.nbl[o] = n;
                    sumB += n;
                }
                nj += __popc(m);
            }
#pragma unroll
            for (int h = 0; h < PLEAF / 32; ++h) {
                const int p = lane + 32 * h;
                if (32 * h >= nA) break;
                const int id = T.leaf_base1 + sA + p;
                int n = 0;
                float w = 0.f;
                if (p < nA) { w = T.c1[id].b.w; n = __float_as_int(T.c1[id].c.z); }
                const bool v = n > 0 && w != 0.f;
                const unsigned m = __ballot_sync(0xffffffffu, v);
                single = single && __all_sync(0xffffffffu, !v || n == 1);
                if (v) { S.ia[na + __popc(m & lt)] = (unsigned char)p; sumA += n; }
                na += __popc(m);
            }
            ++n_tiles;
            if (na == 0 || nj == 0) { __syncwarp(); continue; }
            __syncwarp();
            // Empty leaves after B's last (the first leaf's position, no weight), so that every
            // lane group of a round finds a pair: B's pairs rounded up to a multiple of the groups
            // (32 / rows of them; at most PPAIRS).
            {
                const int njp = (nj + 1) >> 1;
                int lim = 0;
                for (int rest = na; rest > 0; rest -= 32) {
                    const int gr = 32 / min(rest, 32);
                    lim = max(lim, (njp + gr - 1) / gr * gr);
                }
                const float* f0 = reinterpret_cast<const float*>(&S.b[0]);
                const float x = f0[0], y = f0[2], z = f0[4], zh = f0[6];
                __syncwarp();
                for (int o = nj + lane; o < 2 * lim; o += 32) {
                    float* f = reinterpret_cast<float*>(&S.b[o >> 1]) + (o & 1);
                    f[0] = x; f[2] = y; f[4] = z; f[6] = zh;
                    f[8] = f[10] = f[12] = f[14] = 0.f;
                    S.ib[o] = S.ib[0];
                    S.nbl[o] = 0;
                }
            }
            __syncwarp();
            C.na = na; C.nj = nj;
            int ecount = 0;
            const unsigned long long pairs = (unsigned long long)__reduce_add_sync(0xffffffffu, sumA) *
                                             __reduce_add_sync(0xffffffffu, sumB);
            if (cls == 1) {
                float o[1][8];
                unsigned none;
                packed_pairs<GEO, KIND, 1>(T, S, C, lane, o, none, ecount);
                // (the counts go in here, not through tile_bin_out, which needs one to add)
                tile_bin_out(o[0], 1u, C.kref, nq, nb, ledge, fb, np, true, true, lane);
                if (!quick && lane == 0) np[C.kref] += pairs;
                n_sure += (unsigned long long)(na * nj);
            } else if (cls == 2 && single) {
                float o[2][8];
                unsigned cn;
                packed_pairs<GEO, KIND, 2>(T, S, C, lane, o, cn, ecount);
                if (ecount <= PESC) {               // (else packed_slow takes all pairs)
                    const unsigned all = (unsigned)(na * nj - ecount), up = __reduce_add_sync(0xffffffffu, cn);
                    n_sure += all;
                    tile_bin_out(o[0], 1u, C.kref, nq, nb, ledge, fb, np, true, true, lane);
                    tile_bin_out(o[1], 1u, C.kref + 1, nq, nb, ledge, fb, np, true, true, lane);
                    if (!quick && lane == 0) { np[C.kref] += all - up; np[C.kref + 1] += up; }
                }
            } else {
                constexpr int W = hist_rows<KIND>(), RF = 32 * hist_words<KIND>();
                // The counts are 32-bit: a tile of more point pairs is taken pair by pair.
                if (pairs >> 32) ecount = PESC + 1;
                const unsigned before = n_acc;
                for (int w0 = 0; w0 <= span && ecount <= PESC; w0 += W) {
                    const int nr = min(W, span + 1 - w0);
                    float4* h4 = reinterpret_cast<float4*>(hist);
                    for (int z = lane; z < nr * (RF / 4); z += 32) h4[z] = make_float4(0.f, 0.f, 0.f, 0.f);
                    __syncwarp();
                    // (one form with the special steps as a branch in the loop: GG of 10^6 points
                    // 159 ms, two forms 155)
                    if ((GEO == TG_ARC || (GEO == TG_SPHEUC && KIND == TK_GG)) && C.special)
                        packed_hist<GEO, KIND, true>(T, S, C, hist, lane, w0, ecount, n_acc);
                    else
                        packed_hist<GEO, KIND, false>(T, S, C, hist, lane, w0, ecount, n_acc);
                    if (ecount > PESC) { n_acc = before; break; }
                    for (int b = 0; b < nr; ++b) {
                        const float* h = hist + b * RF;
                        const float4 a = reinterpret_cast<const float4*>(h)[lane];
                        float o[8] = {a.x, a.y, a.z, 0.f, 0.f, 0.f, 0.f, 0.f};
                        if constexpr (KIND == TK_GG) {
                            const float4 x = reinterpret_cast<const float4*>(h + 128)[lane];
                            o[3] = x.x; o[4] = x.y; o[5] = x.z; o[6] = x.w;
                        } else if constexpr (KIND == TK_SC) {
                            o[3] = h[128 + lane];
                        }
                        sphere_gg<GEO, KIND>(o);
                        const unsigned cn = __float_as_uint(a.w);
                        tile_bin_out(o, cn, C.kref + w0 + b, nq, nb, ledge, fb, np, quick, true, lane);
                    }
                }
            }
            n_pairs += C.self ? (unsigned long long)(na * (na - 1) / 2) : (unsigned long long)(na * nj);
            if (ecount) {
                __syncwarp();
                const uint2 n = packed_slow(T, S, C.idA, C.idB, na, nj, C.self, ecount > PESC, ecount, fb, np, lane);
                n_acc += n.x;
                n_esc += n.y;
            }
            if (++since_flush >= PFLUSH) {
                since_flush = 0;
                __syncwarp();
                for (int z = lane; z < nq * nb; z += 32) {
                    const float x = fb[z];
                    if (x != 0.f) {
                        float2 f = fd[z];
                        df_add(f, x);
                        fd[z] = f;
                        fb[z] = 0.f;
                    }
                }
            }
            __syncwarp();
        }
    }
    if (since_flush >= 0) {
        __syncwarp();
        for (int z = lane; z < nq * nb; z += 32) {
            float2 f = fd[z];
            df_add(f, fb[z]);
            fd[z] = f;
        }
        __syncwarp();
        double* wa = T.wacc + (size_t)(T.tile_wbase + gw) * nq * nb;
        warp_add_totals(wa, fd, nq * nb, lane);
        unsigned long long* wn = T.wnp + (size_t)(T.tile_wbase + gw) * nb;
        for (int z = lane; z < nb; z += 32) wn[z] += np[z];
        unsigned long long a64 = n_acc, e64 = n_esc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a64 += __shfl_xor_sync(0xffffffffu, a64, o);
            e64 += __shfl_xor_sync(0xffffffffu, e64, o);
        }
        a64 += n_sure;
        if (lane == 0) {
            unsigned long long* w = T.wctr + (size_t)(T.tile_wbase + gw) * 8;
            const unsigned long long o1 = w[1], o4 = w[4], o5 = w[5], o6 = w[6];
            w[1] = o1 + a64;
            w[4] = o4 + n_tiles;
            w[5] = o5 + n_pairs;
            w[6] = o6 + e64;
        }
    }
    if (nt > 0) {
        // The last block empties the tile list for the next expansion launch.
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const unsigned long long prev = atomicAdd(&T.tctl[1], 1ull);
            if (prev == (unsigned long long)gridDim.x - 1) {
                T.tctl[0] = 0ull;
                T.tctl[1] = 0ull;
                __threadfence();
            }
        }
    }
}

struct PackedSet { TileKernel cls, run; size_t warp; };

template <int GEO, int KIND>
PackedSet packed_set(const TravParams& T)
{
    return PackedSet{k_tile_class<GEO>, k_tiles_packed<GEO, KIND>, packed_warp_bytes<KIND>(T.nqf, T.nbins)};
}

template <int GEO>
bool pick_kind(const TravParams& T, PackedSet& K)
{
    if (T.k1 == DN && T.k2 == DN) { K = packed_set<GEO, TK_NN>(T); return true; }
    if (T.k2 != DG) { K = packed_set<GEO, TK_SC>(T); return true; }
    if constexpr (GEO != TG_3D)
        if (T.k1 == DG && T.s1 == 2 && T.s2 == 2) { K = packed_set<GEO, TK_GG>(T); return true; }
    return false;
}

// The kernels for T's classes and geometry; none for the other complex kinds, GG in 3-d and
// brute fields (whose cells' sizes bound nothing): k_tiles takes those.
bool pick(const TravParams& T, PackedSet& K)
{
    if (T.brute || T.nbins > KEY_MAXNB) return false;
    // Squared separations are normal FP32 numbers, and max_sep is the last bin's edge.
    if (!(T.fminsep >= 1e-15f && T.fmaxsep <= 1e15f)) return false;
    if (!(std::fabs(0.5 * std::log(T.maxsepsq / T.minsepsq) - T.nbins * T.binsize) <= 1e-9 * T.binsize)) return false;
    if (T.coords == SPHERE && T.k2 == DG && T.fminsep < 1e-13f) return false;    // (k_tile_class)
    bool found;
    if (T.coords == FLAT) found = pick_kind<TG_FLAT>(T, K);
    else if (T.coords == SPHERE) found = T.metric == ARC ? pick_kind<TG_ARC>(T, K) : pick_kind<TG_SPHEUC>(T, K);
    else found = pick_kind<TG_3D>(T, K);
    return found && K.warp * PW <= 227 * 1024;      // (many bins take the shared memory)
}

}  // namespace

bool packed_tiles(const TravParams& T)
{
    PackedSet K;
    return pick(T, K);
}

int packed_grid(const TravParams& T, int* blocks, int* nwarps)
{
    PackedSet K;
    if (!pick(T, K)) { set_last_error("no packed tile kernel for these classes"); return 1; }
    int dev = 0, nsm = 0, per = 0;
    TC_CU(cudaGetDevice(&dev));
    TC_CU(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const size_t sm = K.warp * PW;
    if (sm > 48 * 1024)
        TC_TRY(allow_smem(K.run, sm));
    TC_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, K.run, PB, sm));
    if (per < 1) per = 1;
    *blocks = nsm * per;
    *nwarps = *blocks * PW;
    return 0;
}

int launch_packed_tiles(const TravParams& T, cudaStream_t st)
{
    PackedSet K;
    pick(T, K);
    count_launch();
    K.cls<<<T.tile_blocks, 256, 0, st>>>(T);
    count_launch();
    K.run<<<T.tile_blocks, PB, K.warp * PW, st>>>(T);
    return 0;
}

}  // namespace tc
