// walk.cu -- the depth-first half of the 2-point traversal (the bin_slop rule on whole
// fields and on patch batches).
//
// The breadth-first expansion (traverse2pt.cu) runs only until its level holds enough items
// to fill the chip many times over.  From there every item is an independent subtree, and
// k_walk takes them in units: a warp takes the next unit from a counter, walks its items
// depth first on a stack of its own and writes the unit's sums to the unit's own row; the
// rows are added up in order at the end.  Which warp walks a unit does not matter to its sums,
// so the results repeat bit for bit although the load is balanced dynamically, without level
// buffers in memory, joins of warp regions, or a launch per chunk.
//
// The decisions are the reference's (BaseCorr2::process11, src/Corr2.cpp:308-389; singleBin,
// include/BinType.h:93-151; CalcSplitSq, include/Split.h:82-101), taken in FP32 with an error
// margin on every comparison.  The squared comparisons of the rule become comparisons of the
// ratio S / r with constants, so that a pair costs one reciprocal and a few compares.  A pair
// inside a margin waits in a list until 32 of them share one pass of the FP64 formulas
// (decide64).
//
// Accepted pairs land mostly in one or two bins while a warp is below one item (the walk
// stays in one item's subtree, whose separations span a few per cent).  Two neighbouring bins
// are therefore summed in registers, per lane; the warp moves them to where its pairs are, and
// pairs of other bins wait in a small list in shared memory that is added by a few lanes at a
// time.  Registers reach the unit's double-float sums every few iterations.
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "tc_internal.cuh"
#include "tc_host.hpp"
#include "traverse2pt.hpp"
#include "pair_math.cuh"
#include "roots.cuh"

namespace tc {

namespace {

constexpr int KB = 128;             // threads of a walk block
constexpr int KW = KB / 32;
// Resident blocks per SM the registers are sized for, measured per class family.  7: 72 registers
// (KK 300K 3-d 9.9 ms; 10.4 with 6).  NN 6: 2M clumped 18.2 ms; 19.0 with 7.  GG 7: 10M 530 ms; 530 with
// 6, 540 with 5, 592 with 4.  The generic projections 5: 96 registers.
constexpr int walk_minb(int kind) { return kind == 3 ? 5 : kind == 0 ? 6 : 7; }
constexpr double W_PER_LN = 2.8853900817779268;    // 2 / ln 2
constexpr int WFLUSH = 32;          // iterations between flushes of the register bins
constexpr int WDRAINS = 8;        // lists added to the FP32 sums between their flushes
// Entries of the list of other bins (at least the 32 that an iteration can add).  64 for the kinds
// of few sums; what GG would gain, its records lose in L1 (10M: 530 ms at 32, 545 at 64).
constexpr int walk_mcap(int kind) { return kind <= 1 ? 64 : 32; }
constexpr int UCAP = 64;            // pairs waiting for the FP64 decision
constexpr int MST = 9;              // words per entry (odd: no bank conflicts)
constexpr unsigned NSMALL = 1u << 21;  // n1 n2 below this is counted in 32 bits between flushes:
                                       // 32 iterations x 32 lanes, or 8 lists of 64, hold it

enum { WG_FLAT = 0, WG_ARC = 1, WG_EUC = 2 };                // geometry (EUC: 3 coordinates)
enum { WK_NN = 0, WK_SC = 1, WK_GG = 2, WK_GEN = 3 };        // class family

// Copies of the FP32 sums of other bins: so many entries of the list are added at once, by 8
// lanes each (an entry is a chain of a load, an addition and a store; one at a time they took a
// sixth of the kernel's instructions).  As many as keep a warp's sums small, and one for GG:
// the shared memory of four is missed as L1 (10M 590 ms, with one 530; KK 300K 3-d 10.7 -> 10.1, NN
// 2M clumped 19.3 -> 18.6).
__host__ __device__ inline int walk_copies(int kind, int nq, int nb)
{ return kind == WK_GG ? 1 : nq * nb <= 128 ? 4 : nq * nb <= 256 ? 2 : 1; }

__host__ __device__ inline size_t walk_warp_bytes(int kind, int nq, int nb)
{
    return ((size_t)nq * nb * 8 + (size_t)nb * 8 + (size_t)walk_copies(kind, nq, nb) * nq * nb * 4 +
            (size_t)nb * 4 + walk_mcap(kind) * MST * 4 + UCAP * 8 + 15) & ~(size_t)15;
}

// The FP64 decision (out of line: about one pair in 3000 takes it).  Returns the action, the
// bin, and r and 2 log2(r / min_sep) of an accepted pair.
__device__ __noinline__ int4 decide_slow(const TravParams& T, int i, int j)
{
    const double dx = T.x1[i] - T.x2[j], dy = T.y1[i] - T.y2[j];
    double dsq = dx * dx + dy * dy;
    if (T.coords != FLAT) { const double dz = T.z1[i] - T.z2[j]; dsq += dz * dz; }
    const Decision D = decide64(T, dsq, (double)T.c1[i].a.w, (double)T.c2[j].a.w);
    const float lg = (float)(((double)D.logr - T.logminsep) * W_PER_LN);
    return make_int4(D.act, D.k, __float_as_int(D.r), __float_as_int(lg));
}

// log2 of a normal x > 0: the exponent apart, and 2 atanh(s) / ln 2, s = (m - 1) / (m + 1), by
// its Taylor series on mantissas m in [sqrt(1/2), sqrt(2)) (|s| < 0.172: the first omitted
// term is below 1e-9).  Within 1e-7 plus one rounding; the hardware logarithm's 2^-22 biases
// the sum of log r of flat catalogs to twice the error of logf.
__device__ __forceinline__ float log2_series(float x)
{
    const int b = __float_as_int(x);
    const int e = (b - 0x3f3504f3) >> 23;
    const float m = __int_as_float(b - (e << 23));
    const float s = __fdividef(m - 1.f, m + 1.f), z = s * s;
    constexpr float c = (float)W_PER_LN;
    const float p = fmaf(z, fmaf(z, fmaf(z, fmaf(z, c / 9.f, c / 7.f), c / 5.f), c / 3.f), c);
    return fmaf(s, p, (float)e);
}

// The correlation products of an accepted pair (DirectHelper, src/Corr2.cpp:394-474), x[0..3].
template <int GEO, int KIND>
__device__ __forceinline__ void walk_products(const TravParams& T, float4 Aa, float4 Ab, float4 Ac, float4 Ba,
                                              float4 Bb, float4 Bc, int i, int j, float dx,
                                              float dy, float dz, float dsq, float r,
                                              float (&x)[4])
{
    if constexpr (KIND == WK_SC) {
        const float wk1 = T.k1 == DN ? Ab.w : Ac.x;
        x[0] = wk1 * Bc.x;                                   // NK, KK
    } else if constexpr (KIND == WK_GG && GEO == WG_FLAT) {
        // ProjectHelper<Flat>: both shears turn by exp(-2i alpha) of r = p2 - p1, so
        // g1 conj(g2) is unchanged and g1 g2 turns by exp(-4i alpha).
        const float inv = __fdividef(1.f, dsq);
        const float er = (dx * dx - dy * dy) * inv, ei = -2.f * dx * dy * inv;
        const float e2r = er * er - ei * ei, e2i = 2.f * er * ei;
        const float pr = Ac.x * Bc.x - Ac.y * Bc.y, pi = Ac.x * Bc.y + Ac.y * Bc.x;
        x[0] = Ac.x * Bc.x + Ac.y * Bc.y;
        x[1] = Ac.y * Bc.x - Ac.x * Bc.y;
        x[2] = pr * e2r - pi * e2i;
        x[3] = pr * e2i + pi * e2r;
    } else if constexpr (KIND == WK_GG) {
        // ProjectHelper<Sphere>, include/ProjectHelper.h:272-388, on accurate differences (see
        // accept_values): directions (sinA, -cosA) at p2 and (-sinA, -cosB) at p1.
        const float sinA = Aa.x * dy - Aa.y * dx;
        const float cosA = fmaf(0.5f * Ba.z, dsq, dz);
        const float cosB = fmaf(0.5f * Aa.z, dsq, -dz);
        const float s2 = sinA * sinA, sp = s2 + POLE_SQ, sm = s2 - POLE_SQ;   // (see POLE_SQ)
        const float i2 = __fdividef(1.f, fmaf(cosA, cosA, sp));
        const float i1 = __fdividef(1.f, fmaf(cosB, cosB, sp));
        const float e2r = fmaf(-cosA, cosA, sm), e2i = 2.f * sinA * cosA;
        const float e1r = fmaf(-cosB, cosB, sm), e1i = -2.f * sinA * cosB;
        const float a2r = (Bc.x * e2r - Bc.y * e2i) * i2, a2i = (Bc.x * e2i + Bc.y * e2r) * i2;
        const float a1r = (Ac.x * e1r - Ac.y * e1i) * i1, a1i = (Ac.x * e1i + Ac.y * e1r) * i1;
        const float rr = a2r * a1r, ri = a2r * a1i, ir = a2i * a1r, ii = a2i * a1i;
        x[0] = rr + ii; x[1] = ri - ir; x[2] = rr - ii; x[3] = ri + ir;
    } else if constexpr (KIND == WK_GEN) {
        TCell P, Q;
        P.a = Aa; P.b = Ab; P.c = Ac; P.d = Ac;
        Q.a = Ba; Q.b = Bb; Q.c = Bc; Q.d = Bc;
        float av[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        unsigned long long nn;
        accept_values(T, P, Q, i, j, dx, dy, dz, dsq, r, 0.f, av, nn);
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = av[3 + q];
    }
}

// Sums v[0..7] over the warp by a reduce-scatter; lanes 4 q hold value q's total.
__device__ __forceinline__ float warp_scatter8(const float (&v)[8], int lane)
{
    float a[4];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float got = __shfl_xor_sync(0xffffffffu, h16 ? v[q] : v[q + 4], 16);
        a[q] = (h16 ? v[q + 4] : v[q]) + got;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float got = __shfl_xor_sync(0xffffffffu, h8 ? a[q] : a[q + 2], 8);
        a[q] = (h8 ? a[q + 2] : a[q]) + got;
    }
    const float got = __shfl_xor_sync(0xffffffffu, h4 ? a[0] : a[1], 4);
    float t = (h4 ? a[1] : a[0]) + got;
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    return t;
}

// acc += the pair's values and c += n where on: predicated adds in place (as a branch, the
// compiler keeps both versions of the sums and moves them between registers, 60 moves per
// iteration).
template <int NQ>
__device__ __forceinline__ void add_if(bool on, float (&acc)[8], unsigned& c, float ww, float r,
                                       float lg, const float (&x)[4], unsigned n)
{
    asm("{.reg .pred p;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "@p add.f32 %0, %0, %5;\n"
        "@p fma.rn.f32 %1, %5, %6, %1;\n"
        "@p fma.rn.f32 %2, %5, %7, %2;\n"
        "@p add.u32 %3, %3, %8;}"
        : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+r"(c)
        : "r"((unsigned)on), "f"(ww), "f"(r), "f"(lg), "r"(n));
    if constexpr (NQ == 4)
        asm("{.reg .pred p;\n"
            "setp.ne.u32 p, %1, 0;\n"
            "@p add.f32 %0, %0, %2;}"
            : "+f"(acc[3]) : "r"((unsigned)on), "f"(x[0]));
    if constexpr (NQ == 7)
        asm("{.reg .pred p;\n"
            "setp.ne.u32 p, %4, 0;\n"
            "@p add.f32 %0, %0, %5;\n"
            "@p add.f32 %1, %1, %6;\n"
            "@p add.f32 %2, %2, %7;\n"
            "@p add.f32 %3, %3, %8;}"
            : "+f"(acc[3]), "+f"(acc[4]), "+f"(acc[5]), "+f"(acc[6])
            : "r"((unsigned)on), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]));
}

// Half a record (32 bytes, so one sector) in one load: the lanes' records lie in different
// lines, and a load costs the L1 a cycle or so per line whatever it takes from it.
__device__ __forceinline__ void load_half(const float4* p, float4& u, float4& v)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(u.x), "=f"(u.y), "=f"(u.z), "=f"(u.w), "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p));
}

__device__ __forceinline__ void df_accumulate(float2* fd, float x)
{
    float2 f = *fd;
    df_add(f, x);
    const float t = f.x + f.y;          // renormalise (|lo| <= ulp(hi) / 2)
    f.y -= t - f.x;
    f.x = t;
    *fd = f;
}

}  // namespace

// Bound: instruction issue (the records of a subtree's cells stay in L1 and L2).
// 557 instructions per 32 evaluations of GG on the sphere, where the expansion kernel, with one
// code path for all classes and interval arithmetic around every comparison, takes 1030.
// Measured, traversal of whole calls, expansion alone -> with the walk: GG 10M points on the
// sphere, bin_slop 0.1, 1058 -> 490 ms; GG 200K flat, bin_slop 1, 15 -> 1.7; KK 300K 3-d
// 72 -> 8.3; NN 2M clumped 46 -> 14; NG 100K x 2M 11.6 -> 5.3; 40 patches of 1M 58 -> 16.5.
// Variants: popping the next 32 items early with a prefetch of their records (+8%, two
// interleaved subtrees share their bins less well); the FP64 decision inside the loop (+10%,
// its call spills the loop's registers); sums under if / else (+5%, see add_if).
template <int GEO, int KIND, bool PATCH>
__global__ void __launch_bounds__(KB, walk_minb(KIND)) k_walk(const __grid_constant__ TravParams T,
                                                        const __grid_constant__ WalkParams W)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NQ = KIND == WK_NN ? 3 : KIND == WK_SC ? 4 : 7;   // values kept per bin
    constexpr int MCAP = walk_mcap(KIND);
    static_assert(MCAP >= 32, "");
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nq = T.nqf, nb = T.nbins;      // nq <= NQ
    unsigned char* wb = smem + wib * walk_warp_bytes(KIND, nq, nb);
    int2* ub = reinterpret_cast<int2*>(wb);                     // pairs for the FP64 decision
    float2* fd = reinterpret_cast<float2*>(ub + UCAP);          // the unit's sums
    unsigned long long* np = reinterpret_cast<unsigned long long*>(fd + nq * nb);
    float* fb = reinterpret_cast<float*>(np + nb);              // FP32 sums of other bins
    const int copies = walk_copies(KIND, nq, nb), fbs = nq * nb;      // (their copies, fbs apart)
    unsigned* nb32 = reinterpret_cast<unsigned*>(fb + copies * fbs); // their pairs, in 32 bits
    float* ml = reinterpret_cast<float*>(nb32 + nb);            // list of other bins' pairs
    int2* stk = W.stacks + (size_t)(blockIdx.x * KW + wib) * W.stack_cap;
    const unsigned lt = (1u << lane) - 1u;

    float acc0[8], acc1[8];                  // register bins K0 and K0 + 1
    unsigned c0 = 0, c1 = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) { acc0[q] = 0.f; acc1[q] = 0.f; }
    int K0 = -4, mcount = 0, drains = 0, since = 0;

    auto flush_regs = [&]() {
        if (K0 >= 0) {
            const float t0 = warp_scatter8(acc0, lane), t1 = warp_scatter8(acc1, lane);
            const unsigned s0 = __reduce_add_sync(0xffffffffu, c0);
            const unsigned s1 = __reduce_add_sync(0xffffffffu, c1);
            const int q = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
            const int kb = K0 + (lane & 1);
            if (q < nq && (lane & 2) == 0 && kb < nb)
                df_accumulate(fd + q * nb + kb, (lane & 1) ? t1 : t0);
            if (lane < 2 && kb < nb) np[kb] += lane ? s1 : s0;
            __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) { acc0[q] = 0.f; acc1[q] = 0.f; }
        c0 = 0; c1 = 0; since = 0;
    };
    auto flush_fb = [&]() {
        for (int q = lane; q < fbs; q += 32) {
            float x = fb[q];
            fb[q] = 0.f;
            for (int c = 1; c < copies; ++c) { x += fb[c * fbs + q]; fb[c * fbs + q] = 0.f; }
            if (x != 0.f) df_accumulate(fd + q, x);
        }
        for (int q = lane; q < nb; q += 32) { np[q] += nb32[q]; nb32[q] = 0u; }
        __syncwarp();
        drains = 0;
    };
    auto drain = [&]() {
        __syncwarp();
        const int q = lane & 7, g = lane >> 3;
        if (q < nq && g < copies) {
            float* my = fb + g * fbs + q * nb;
#pragma unroll 2
            for (int t = g; t < mcount; t += copies) {
                const float* e = ml + t * MST;
                my[__float_as_int(e[7])] += e[q];
            }
        }
        mcount = 0;
        __syncwarp();
        if (++drains == WDRAINS) flush_fb();
    };

    for (int guard = 0; guard < (1 << 30); ++guard) {
        // The next unit: items first, first + step, ... below count of its segment's list.
        unsigned u = 0;
        if (lane == 0) u = (unsigned)atomicAdd(W.next, 1ull);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= W.n_units) break;
        unsigned it = u, step = W.n_units, count = W.n_items;
        int pair = 0;
        if (PATCH) {
            int lo = 0, hi = T.npair;          // unit_off[lo] <= u < unit_off[hi]
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (W.unit_off[mid] <= (int)u) lo = mid; else hi = mid;
            }
            pair = lo;
            it = u - W.unit_off[lo];
            step = W.unit_off[lo + 1] - W.unit_off[lo];
            count = (unsigned)(T.proot_off[lo + 1] - T.proot_off[lo]);
        }
        for (int q = lane; q < nq * nb; q += 32) fd[q] = make_float2(0.f, 0.f);
        for (int q = lane; q < copies * fbs; q += 32) fb[q] = 0.f;
        for (int q = lane; q < nb; q += 32) { np[q] = 0ull; nb32[q] = 0u; }
        __syncwarp();
        unsigned n_eval = 0, n_acc = 0, n_esc = 0;   // of the unit
        unsigned long long n_eval64 = 0, n_acc64 = 0;
        K0 = -4;
        int sp = 0, ucount = 0;
        while (true) {
            // Items: pairs that wait for the FP64 decision (when 32 of them do, or nothing else is
            // left: all lanes then share its cost), the top of the stack, or the unit's next 32.
            int2 task = make_int2(0, 0);
            int4 slow = make_int4(-1, 0, 0, 0);     // the FP64 decision of this lane's pair
            int nt;
            if (ucount >= 32 || (sp == 0 && ucount > 0)) {
                nt = min(ucount, 32);
                ucount -= nt;
                if (lane < nt) {
                    task = ub[ucount + lane];
                    slow = decide_slow(T, task.x, task.y);
                }
                __syncwarp();
                n_esc += nt;
                n_eval -= nt;                       // (counted when first taken)
            } else if (sp > 0) {
                nt = min(sp, 32);
                sp -= nt;
                if (lane < nt) task = stk[sp + lane];
            } else {
                if (it >= count) break;
                const unsigned long long g = it + (unsigned long long)lane * step;
                const bool ok = g < count;
                if (ok) task = PATCH ? make_pair_root(T, pair, (long long)g)
                                     : (W.items ? W.items[g] : make_root(T, (long long)g));
                nt = __popc(__ballot_sync(0xffffffffu, ok));   // (the first lanes)
                const unsigned long long nx = it + 32ull * step;
                it = nx < count ? (unsigned)nx : count;
            }
            const bool has = lane < nt;
            n_eval += nt;
            if (sp + 128 > W.stack_cap) {       // (the host then takes the expansion instead)
                if (lane == 0) atomicCAS(T.err, 0, DEV_STACK_OVERFLOW);
                it = count;
                sp = 0;
                ucount = 0;
                continue;
            }
            // Both records, without branches: a self item (j < 0) reads its cell twice, an idle
            // lane cell 0.
            const int i = task.x, j = task.y;
            const bool self = j < 0;
            const TCell* A = T.c1 + i;
            const TCell* B = self ? A : T.c2 + j;
            float4 Aa, Ab, Ac, Ad, Ba, Bb, Bc, Bd;
            load_half(&A->a, Aa, Ab);
            load_half(&B->a, Ba, Bb);
            load_half(&A->c, Ac, Ad);
            load_half(&B->c, Bc, Bd);
            const bool live = has && Ab.w != 0.f && Bb.w != 0.f;
            const float dx = (Aa.x - Ba.x) + (Ab.x - Bb.x);
            const float dy = (Aa.y - Ba.y) + (Ab.y - Bb.y);
            const float dz = GEO == WG_FLAT ? 0.f : (Aa.z - Ba.z) + (Ab.z - Bb.z);
            const float dsq = GEO == WG_FLAT ? fmaf(dx, dx, dy * dy)
                                             : fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            // r = sqrt(dsq): the approximate reciprocal root and one Heron step.
            const float y = rsqrtf(dsq);
            float r = dsq * y;
            r = fmaf(0.5f * y, fmaf(-r, r, dsq), r);
            if (dsq == 0.f) r = 0.f;
            if (GEO == WG_ARC) {                // arc_from_chord_sq on the chord
                const float h = 0.5f * r, h2 = h * h;
                const float ser = r * fmaf(h2, fmaf(h2, fmaf(h2, 5.f / 112.f, 3.f / 40.f), 1.f / 6.f), 1.f);
                const bool wide = r >= 0.25f;
                r = ser;
                if (__any_sync(0xffffffffu, wide)) { if (wide) r = 2.f * asinf(h); }
            }
            // The decision (see the head of the file).  Every flag is a certain statement: the
            // error bounds are r 2.5e-6, S and f 3.2e-6 relative, kk ek absolute, and the
            // constants carry margins of 6e-6; a pair without a certain outcome (or a NaN)
            // goes to the FP64 formulas.
            const float s1 = Aa.w, s2 = Ba.w;
            const float S = s1 + s2, rpS = r + S, rmS = r - S;
            const float rinv = __fdividef(1.f, r);
            const float f = S * rinv;
            // singleBin, include/BinType.h:93-151.
            float lg = log2_series(r * r * T.finvminsepsq);           // 2 log2(r / min_sep)
            const float kk = lg * W.per_log2;
            const float ek = fmaf(fabsf(lg), W.ek1, W.ek0);
            // int(kk) truncates toward zero, as in the reference (kk < 0 is possible).
            const float ik = truncf(kk), fr = kk - ik;
            const bool clear = fabsf(fabsf(fr) - 0.5f) <= 0.5f - ek;   // the bin is certain
            const float t4 = fabsf(fmaf(fminf(fr, 1.f - fr), T.fbinsize, T.fb));
            const float t5 = fabsf(fmaf(fr, T.fbinsize, T.fb) - f * f);
            const float tt = fminf(t4, t5);
            const float mm = fmaf(ek, T.fbinsize, fmaf(f, 1.4e-5f, W.t0));
            // Below b (or a point pair) one bin; above a or h more than one; between b and h by
            // the place in the bin.
            const bool passA = f < W.a_lo, overB = f > W.b_hi;
            const bool mid = passA && overB && f < W.h_lo && clear;
            const bool one = S == 0.f || (passA && f < W.b_lo) || (mid && f < tt - mm);
            bool split = S > 0.f && (f > W.a_hi || (passA && overB && f > W.h_hi) ||
                                     (mid && f > tt + mm));
            int k = (int)ik;
            bool accept = one && clear;
            // CalcSplitSq, include/Split.h:82-101.
            bool sw = s2 > s1;
            const float big = fmaxf(s1, s2), sml = fminf(s1, s2), g = sml * rinv;
            const bool lone = big > 2.f * sml;
            bool both = !lone && g > W.c_hi;
            bool sure = accept || (split && (lone || both || g < W.c_lo));
            const bool cand = live && !self;
            if (__any_sync(0xffffffffu, cand && !(rmS > W.min_hi && rpS < W.max_lo))) {
                // Some pair is near an end of the range: tooSmallDist and tooLargeDist
                // (include/BinType.h:70-82: r + S < min_sep, r - S >= max_sep), isRSqInRange
                // (61-66), the clamp of directProcess11.
                const float e = 6e-6f * rpS;
                const bool drop = rpS < W.min_lo || rmS >= T.fmaxsep + e;
                const bool near = rpS > W.min_hi && rmS < T.fmaxsep - e;
                const bool out = one && (r < W.min_lo || r > W.max_hi);
                if (k == T.nbins) k = T.nbins - 1;
                accept = accept && r > W.min_hi && r < W.max_lo;
                sure = drop || (near && (accept || out || (split && sure)));
                accept = accept && !drop;
                split = split && !drop;
            }
            const bool inb = (unsigned)k < (unsigned)T.nbins;
            sure = sure && (inb || !accept);
            const unsigned mslow = __ballot_sync(0xffffffffu, cand && !sure && slow.x < 0);
            accept = accept && cand && sure;
            split = split && cand && sure;
            if (mslow) {
                if (mslow & (1u << lane)) ub[ucount + __popc(mslow & lt)] = task;
                ucount += __popc(mslow);
                __syncwarp();
            }
            if (slow.x >= 0) {
                accept = slow.x == ACT_ACCEPT;
                split = slow.x >= ACT_SPLIT1;
                both = slow.x == ACT_SPLIT12;
                sw = slow.x == ACT_SPLIT2;
                if (accept) { k = slow.y; r = __int_as_float(slow.z); lg = __int_as_float(slow.w); }
            }
            // process2, src/Corr2.cpp:290-306: a self item of size above min_sep / 2.
            bool down = self && live && !(s1 <= W.half_min);
            const bool s1st = down || both || !sw, s2nd = !down && (both || sw);
            if ((split || down) && ((s1st && __float_as_int(Ac.w) < 0) ||
                                    (s2nd && __float_as_int(Bc.w) < 0))) {
                atomicCAS(T.err, 0, DEV_BAD_CHILD);     // (a validated tree has none)
                split = down = false;
            }

            // Accepted pairs: the register bins follow them.
            const int kacc = accept ? k : -1;
            const unsigned ma = __ballot_sync(0xffffffffu, accept);
            if (ma) {
                n_acc += __popc(ma);
                unsigned mh = __ballot_sync(0xffffffffu, accept && (unsigned)(k - K0) < 2u);
                int kn = K0;
                if (2 * __popc(mh) < __popc(ma)) {
                    // Most pairs lie elsewhere: move the register bins to where one of them is,
                    // if they cover more of these pairs there.
                    const int kf = __shfl_sync(0xffffffffu, kacc, __ffs(ma & ~mh) - 1);
                    const unsigned me = __ballot_sync(0xffffffffu, kacc == kf);
                    const unsigned md = __ballot_sync(0xffffffffu, accept && kacc == kf - 1);
                    const unsigned mu = __ballot_sync(0xffffffffu, kacc == kf + 1);
                    const bool low = __popc(md) > __popc(mu);
                    const unsigned mn = me | (low ? md : mu);
                    if (__popc(mn) > __popc(mh) + 4 || K0 < 0) {
                        kn = low ? kf - 1 : kf;
                        mh = mn;
                    }
                }
                if (kn != K0 || since >= WFLUSH) {
                    flush_regs();
                    K0 = kn;
                }
                ++since;
                const unsigned mmiss = ma & ~mh;
                if (mcount + __popc(mmiss) > MCAP) drain();
                // The pair's values, on every lane (a lane without a pair adds none of them).
                const float ww = Ab.w * Bb.w;
                float x[4] = {0.f, 0.f, 0.f, 0.f};
                if (KIND != WK_GEN || accept)
                    walk_products<GEO, KIND>(T, Aa, Ab, Ac, Ba, Bb, Bc, i, j, dx, dy, dz, dsq, r, x);
                const unsigned n1 = (unsigned)__float_as_int(Ac.z), n2 = (unsigned)__float_as_int(Bc.z);
                unsigned ns = n1 * n2;
                const bool many = (__umulhi(n1, n2) | (ns / NSMALL)) != 0u;
                if (__any_sync(0xffffffffu, accept && many)) {
                    if (accept && many) atomicAdd(&np[k], (unsigned long long)n1 * n2);
                    if (many) ns = 0u;
                }
                add_if<NQ>(accept && k == K0, acc0, c0, ww, r, lg, x, ns);
                add_if<NQ>(accept && k == K0 + 1, acc1, c1, ww, r, lg, x, ns);
                if (mmiss & (1u << lane)) {
                    float* o = ml + (mcount + __popc(mmiss & lt)) * MST;
                    o[0] = ww; o[1] = ww * r; o[2] = ww * lg;
#pragma unroll
                    for (int q = 3; q < NQ; ++q) o[q] = x[q - 3];
                    o[7] = __int_as_float(k);
                    if (ns) atomicAdd(&nb32[k], ns);
                }
                mcount += __popc(mmiss);
            }
            // Children: 2 or 4 per split pair, 3 per self item.
            const unsigned m2 = __ballot_sync(0xffffffffu, split || down);
            if (m2) {
                const unsigned m3 = __ballot_sync(0xffffffffu, down);
                const unsigned m4 = __ballot_sync(0xffffffffu, split && both);
                if (split || down) {
                    const int l1 = s1st ? __float_as_int(Ac.w) : i;
                    const int r1 = s1st ? __float_as_int(Ad.x) : i;
                    const int l2 = s2nd ? __float_as_int(Bc.w) : j;
                    const int r2 = s2nd ? __float_as_int(Bd.x) : j;
                    int2* o = stk + sp + 2 * __popc(m2 & lt) + __popc(m3 & lt) + 2 * __popc(m4 & lt);
                    o[0] = make_int2(l1, down ? -1 : l2);
                    o[1] = make_int2(r1, down ? -1 : r2);
                    if (down || both) o[2] = make_int2(l1, down ? r1 : r2);
                    if (both && !down) o[3] = make_int2(r1, l2);
                }
                sp += 2 * __popc(m2) + __popc(m3) + 2 * __popc(m4);
                __syncwarp();
            }
            if (n_eval >= (1u << 31)) { n_eval64 += n_eval; n_acc64 += n_acc; n_eval = 0; n_acc = 0; }
        }
        if (n_acc64 + n_acc) {
            flush_regs();
            drain();
            flush_fb();
            double* row = W.rows + (size_t)u * nq * nb;
            // Quantity 2 was gathered as w w 2 log2(r / min_sep): the constants of log r come in
            // here, in FP64 (as FP32 factors they would bias its sum by some 1e-8).
            for (int q = lane; q < nq * nb; q += 32) {
                double v = df_value(fd[q]);
                if (q >= 2 * nb && q < 3 * nb)
                    v = v * (1. / W_PER_LN) + T.logminsep * df_value(fd[q - 2 * nb]);
                row[q] = v;
            }
            unsigned long long* rn = W.rownp + (size_t)u * nb;
            for (int q = lane; q < nb; q += 32) rn[q] = np[q];
        }
        if (lane == 0) {
            atomicAdd(&T.counters[0], n_eval64 + n_eval);
            if (n_acc64 + n_acc) atomicAdd(&T.counters[1], n_acc64 + n_acc);
            if (n_esc) atomicAdd(&T.counters[2], (unsigned long long)n_esc);
        }
        __syncwarp();
    }
}

// Sums of a list of rows (nd doubles and ni u64 each) per segment: segment s of off, or slice
// s of gridDim.x equal slices.  RY threads share a column, every RY-th row each, and are added
// in order, so the sums do not depend on timing.
constexpr int RX = 32, RY = 8;

__global__ void __launch_bounds__(RX * RY) k_sum_rows(const double* rows,
                                                      const unsigned long long* rownp,
                                                      long long nrow, const int* off, int nd,
                                                      int ni, double* out,
                                                      unsigned long long* outnp)
{
    __shared__ double shd[RY][RX];
    __shared__ unsigned long long shi[RY][RX];
    const int tx = threadIdx.x % RX, ty = threadIdx.x / RX;
    const int c = blockIdx.y * RX + tx;
    const long long nsl = gridDim.x, s = blockIdx.x;
    const long long r0 = off ? off[s] : nrow * s / nsl, r1 = off ? off[s + 1] : nrow * (s + 1) / nsl;
    double t = 0.;
    unsigned long long n = 0;
    if (c < nd) {
#pragma unroll 8
        for (long long r = r0 + ty; r < r1; r += RY) t += rows[(size_t)r * nd + c];
    } else if (c < nd + ni) {
#pragma unroll 8
        for (long long r = r0 + ty; r < r1; r += RY) n += rownp[(size_t)r * ni + (c - nd)];
    }
    shd[ty][tx] = t;
    shi[ty][tx] = n;
    __syncthreads();
    if (ty == 0) {
        for (int q = 1; q < RY; ++q) { t += shd[q][tx]; n += shi[q][tx]; }
        if (c < nd) out[(size_t)s * nd + c] = t;
        else if (c < nd + ni) outnp[(size_t)s * ni + (c - nd)] = n;
    }
}

namespace {

using WalkKernel = void (*)(TravParams, WalkParams);

int walk_kind(const TravParams& T)
{
    if (T.k1 == DN && T.k2 == DN) return WK_NN;
    if (T.k2 != DG) return WK_SC;
    const bool euc = T.coords != FLAT && T.metric != ARC;
    return !euc && T.k1 == DG && T.s1 == 2 && T.s2 == 2 ? WK_GG : WK_GEN;
}

template <int GEO, bool PATCH>
WalkKernel pick_kind(const TravParams& T)
{
    switch (walk_kind(T)) {
      case WK_NN: return k_walk<GEO, WK_NN, PATCH>;
      case WK_SC: return k_walk<GEO, WK_SC, PATCH>;
      case WK_GG: return k_walk<GEO, GEO == WG_EUC ? WK_GEN : WK_GG, PATCH>;
      default: return k_walk<GEO, WK_GEN, PATCH>;
    }
}

template <bool PATCH>
WalkKernel pick(const TravParams& T)
{
    if (T.coords == FLAT) return pick_kind<WG_FLAT, PATCH>(T);
    if (T.metric == ARC) return pick_kind<WG_ARC, PATCH>(T);
    return pick_kind<WG_EUC, PATCH>(T);
}

WalkKernel pick(const TravParams& T) { return T.mode == 3 ? pick<true>(T) : pick<false>(T); }

}  // namespace

void walk_constants(const TravParams& T, WalkParams& W)
{
    // Margins on each constant: both sides' errors and the constant's own rounding (6e-8) stay below
    // 6e-6.  dsq is within 5e-7 of itself (two roundings per coordinate difference, the squares and
    // their sum; the records' low parts add 4e-15 of the coordinates), r within 6e-7 (the Heron
    // step 1.2e-7, an arc's series or asinf 3e-7): 2.5e-6 is allowed.  S = s1 + s2 is one rounding
    // of exact sizes, S / r and the smaller size / r a reciprocal (2 ulps) and a product more: 3.2e-6
    // is allowed.
    const double m = 6e-6;
    const double a = T.a, b = T.b, h = 0.5 * (T.binsize + T.b);
    const double c = std::sqrt(0.3422) * std::fmin(std::fabs(a), std::fabs(b));
    auto lo = [&](double v) { return (float)(v * (1. - m)); };
    auto hi = [&](double v) { return (float)(v * (1. + m)); };
    W.min_lo = lo(T.minsep); W.min_hi = hi(T.minsep);
    W.max_lo = lo(T.maxsep); W.max_hi = hi(T.maxsep);
    W.a_lo = lo(a); W.a_hi = hi(a); W.b_lo = lo(b); W.b_hi = hi(b);
    W.h_lo = lo(h); W.h_hi = hi(h); W.c_lo = lo(c); W.c_hi = hi(c);
    // kk's error: ln r's 2.5e-6, the logarithm's 1e-7 and the roundings' 3e-7
    // (1 + |lr|), in bins.
    W.per_log2 = (float)(1. / (W_PER_LN * T.binsize));
    W.ek0 = (float)((2.5e-6 + 4e-7) / T.binsize + 1e-6);
    W.ek1 = (float)(3e-7 / (W_PER_LN * T.binsize));
    W.t0 = (float)(3e-7 * (T.binsize + T.b));
    // The largest float not above min_sep / 2: the reference compares the float size with the
    // double.
    W.half_min = (float)T.halfminsep;
    if ((double)W.half_min > T.halfminsep) W.half_min = std::nextafter(W.half_min, 0.f);
}

int walk_grid(const TravParams& T, int* blocks, int* nwarps)
{
    int dev = 0, nsm = 0, per = 0;
    TC_CU(cudaGetDevice(&dev));
    TC_CU(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const size_t sm = walk_warp_bytes(walk_kind(T), T.nqf, T.nbins) * KW;
    const WalkKernel k = pick(T);
    if (sm > 48 * 1024)
        TC_TRY(allow_smem(k, sm));
    TC_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, KB, sm));
    if (per < 1) per = 1;
    *blocks = nsm * per;
    *nwarps = *blocks * KW;
    return 0;
}

int launch_walk(const TravParams& T, const WalkParams& W, int blocks, cudaStream_t st)
{
    const size_t sm = walk_warp_bytes(walk_kind(T), T.nqf, T.nbins) * KW;
    count_launch();
    pick(T)<<<blocks, KB, sm, st>>>(T, W);
    TC_CU(cudaGetLastError());
    return 0;
}

int launch_sum_rows(const double* rows, const unsigned long long* rownp, long long nrow,
                    const int* off, int nseg, int nd, int ni, double* out,
                    unsigned long long* outnp, cudaStream_t st)
{
    count_launch();
    k_sum_rows<<<dim3((unsigned)nseg, (unsigned)((nd + ni + RX - 1) / RX)), RX * RY, 0, st>>>(
        rows, rownp, nrow, off, nd, ni, out, outnp);
    TC_CU(cudaGetLastError());
    return 0;
}

int sum_rows_preload()
{
    cudaFuncAttributes at;
    TC_CU(cudaFuncGetAttributes(&at, k_sum_rows));
    return 0;
}

}  // namespace tc
