// zeta.cu -- the batched Zeta contraction over vertex records (calculateZeta,
// src/Corr3.cpp:1861-2087; MultipoleHelper<1..6>::CalculateZeta, 2108-3082).
//
// For every n and every entry (a, b) of the nbins x nbins matrix
//   gam0 += (wg1 G_a[n-1]) G_b[-n-1]        gam1 += (conj(wg1) G_a[n+1]) G_b[-n+1]
//   gam2 += (wg1 G_a[n-1]) conj(G_b[n+1])   gam3 += (wg1 conj(G_a[-n+1])) G_b[-n-1]
//   weight += (w1 W_a[n]) conj(W_b[n])
// over the records whose row range [ks, mk) holds min(a, b): a sum of outer products over
// vertices.  These are GGG's sums (MultipoleHelper<5>).  With shift 0 the G indices are n and -n
// and wg1 is the real w1 or w1 k1 of an N or K vertex, which makes gam0 and gam2 NGG's / KGG's
// zeta0 and zeta1 (MultipoleHelper<2>, src/Corr3.cpp:2216-2405).
//
//   * Only n >= 0 is contracted: exchanging the factors, gam0, gam1 and weight of (a, b, -n) are
//     those of (b, a, n), and gam2 of (a, b, -n) is gam3 of (b, a, n) (k_mp_reduce reads them so).
//   * The records are put in the order of their row ranges (a counting sort of their offsets)
//     and cut into segments of one range each.  Within a segment the set of entries is fixed:
//     its 4 x 2 tiles are dealt out to the threads, the sums run over the records without any
//     test, and the range is applied when they are added up.  At 20 bins and 500,000 points a
//     record has 101 of the 400 entries on average, 134 with the ragged tiles.
//   * A thread keeps its tile's 80 sums in registers, over 256 records at most, 40 with more than 32 bins
//     (FP32); then they go to FP64.  A block's threads are S streams of the segment's tiles, each with
//     every S-th record.  The five columns of a chunk of records are loaded into registers while
//     the chunk before is contracted from shared memory.
//
// Bounds: 98e9 FP32 multiply-adds of needed entries (131e9 with the tiles' edges, 3.5 ms at the
// FMA rate) and 17 GB of records (2.5 ms of measured copy bandwidth) at 500,000 points, 20 bins,
// max_n 30; measured 19.8 ms for the contraction and 0.4 ms for the ordering.  Before, a tcgen05
// kernel took 172 ms: it did every record's full matrix for all n of both signs, twice (the row
// range as a difference of two), on 3 x TF32 operands whose staging (shared-memory stores)
// bound it, and its TMEM sums were the least precise of the path: the error of the whole
// correlation against FP64 falls from 2.6e-6 to 5.4e-7 (5,000 points, 10 bins, max_n 12).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "tc_internal.cuh"
#include "tc_host.hpp"
#include "multipole.hpp"

namespace tc {

namespace {

constexpr int ZT = 192;             // threads per contraction block
constexpr int ZIT = 2;              // (record, bin) items a thread loads per chunk
constexpr int ZPAD = 4;             // bins a ragged tile may read past the last record
// Records of a segment.  Up to 32 bins a stream adds up 64 to 256 of them in FP32 (256 is a segment of
// one stream); with more bins every segment is of one or two streams, and runs of 256 were less
// precise than the two levels of some 30 and 16 records that were summed there before:
// against FP64, 5000 points, 40 bins 8.4e-7 and 6.6e-7, 64 bins 1.6e-6 and 1.1e-6 of zeta's
// largest value.  Runs of 40: see RUN_MANY.
constexpr int SEG_MIN = 256, SEG_MAX = 4096, RUN = 64, RUN_MANY = 40, MANY_BINS = 32;

__device__ __forceinline__ int record_key(const ZParams& Q, unsigned off)
{
    if (off == ZOFF_NONE) return -1;
    const float* R = Q.rec + 4 * (size_t)off;
    return __float_as_int(R[1]) * (Q.nbd + 1) + __float_as_int(R[2]);
}

// Row range counts, then (scatter) the records' offsets in the order of their ranges.
__global__ void __launch_bounds__(256) k_zrows(ZParams Q, bool scatter)
{
    const int lane = threadIdx.x & 31;
    for (long long i0 = (long long)blockIdx.x * 256 + threadIdx.x - lane; i0 < Q.nrec;
         i0 += (long long)gridDim.x * 256) {
        const long long i = i0 + lane;
        const unsigned off = i < Q.nrec ? Q.off[i] : ZOFF_NONE;
        const int key = record_key(Q, off);
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if (lane == leader && key >= 0)
            base = atomicAdd((scatter ? Q.first : Q.count) + key, __popc(peers));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (scatter && key >= 0) Q.order[base + __popc(peers & ((1u << lane) - 1u))] = off;
    }
}

// first[key]: the place of the key's first record; the segments of all keys.  A segment gives
// each stream of its tiles RUN or RUN_MANY records, so that adding up 80 sums per thread stays small.
__global__ void __launch_bounds__(1024) k_zrows_segments(ZParams Q)
{
    __shared__ int wsum[2][32];
    __shared__ int tot[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nkey = Q.nbd * (Q.nbd + 1);
    int rec0 = 0, seg0 = 0;
    for (int k0 = 0; k0 < nkey; k0 += 1024) {
        const int key = k0 + tid;
        const int c = key < nkey ? Q.count[key] : 0;
        const int ks = key / (Q.nbd + 1), mk = key - ks * (Q.nbd + 1);
        const int f = Q.nbins / Q.nbd;      // 2 for a three-field cross, else 1
        const int ent = f * f * ((Q.nbd - ks) * (Q.nbd - ks) - (Q.nbd - mk) * (Q.nbd - mk));
        const int streams = max(1, ZT * 6 / max(ent, 6));
        const int len = Q.nbins > MANY_BINS ? min(RUN_MANY * streams, SEG_MAX)
                                            : min(max(RUN * streams, SEG_MIN), SEG_MAX);
        const int ns = (c + len - 1) / len;
        int x = c, y = ns;
        for (int o = 1; o < 32; o <<= 1) {
            const int px = __shfl_up_sync(0xffffffffu, x, o), py = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) { x += px; y += py; }
        }
        if (lane == 31) { wsum[0][wid] = x; wsum[1][wid] = y; }
        __syncthreads();
        int bx = rec0, by = seg0;
        for (int w = 0; w < wid; ++w) { bx += wsum[0][w]; by += wsum[1][w]; }
        if (tid == 1023) { tot[0] = bx + x; tot[1] = by + y; }
        bx += x - c;
        by += y - ns;
        if (key < nkey) Q.first[key] = bx;
        for (int s = 0; s < ns; ++s)
            Q.segs[by + s] = make_int4(bx + s * len, min(len, c - s * len), ks, mk);
        __syncthreads();
        rec0 = tot[0];
        seg0 = tot[1];
    }
    if (tid == 0) { *Q.nseg = seg0; Q.first[nkey] = rec0; }
}

__global__ void __launch_bounds__(ZT, 2) k_mp_zeta(ZParams Q)
{
    extern __shared__ float4 zsh[];     // [buffer][A0 A1, A3 AW, B0 B1, B2 BW][record][bin]
    __shared__ int list_sh[ZT], wsum_sh[ZT / 32];
    const int nb = Q.nbins, nbd = Q.nbd, M = Q.maxn, gst = 2 * M + 3, sh = Q.shift;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int tcols = (nb + 1) >> 1, ntile = ((nb + 3) >> 2) * tcols;
    const int ntc = (ntile + ZT - 1) / ZT;          // a segment may have several lists of tiles
    const int chunk = min(64, max(1, ZIT * ZT / nb));
    const int comp = chunk * nb + ZPAD;             // float4 per component
    const long long items = (long long)*Q.nseg * (M + 1) * ntc;
    // Consecutive items are the n of one segment: its records stay in L2.
    for (long long item = blockIdx.x; item < items; item += gridDim.x) {
        const long long seg = item / ((M + 1) * ntc);
        const int rest = (int)(item - seg * ((M + 1) * ntc));
        const int n = rest / ntc, tc = rest - n * ntc;
        const int4 sg = Q.segs[seg];
        const int ks = sg.z, mk = sg.w;
        const int col0 = nbd == nb ? ks : 0, ncol = nb - col0;      // the record's columns
        // The segment's tiles (those with an entry in the row range), ZT of them from ZT tc.
        int nvalid = 0;
        __syncthreads();
        for (int t0 = 0; t0 < ntile; t0 += ZT) {
            const int t = t0 + tid;
            bool ok = false;
            if (t < ntile) {
                const int a0 = 4 * (t / tcols), b0 = 2 * (t % tcols);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int a = a0 + (e >> 1), b = b0 + (e & 1);
                    const int m = min(a >= nbd ? a - nbd : a, b >= nbd ? b - nbd : b);
                    ok = ok || (a < nb && b < nb && m >= ks && m < mk);
                }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, ok);
            if (lane == 0) wsum_sh[wid] = __popc(bal);
            __syncthreads();
            int rank = nvalid + __popc(bal & ((1u << lane) - 1u)) - tc * ZT;
            for (int w = 0; w < ZT / 32; ++w) {
                if (w < wid) rank += wsum_sh[w];
                nvalid += wsum_sh[w];
            }
            if (ok && rank >= 0 && rank < ZT) list_sh[rank] = t;
            __syncthreads();
        }
        const int nv = min(ZT, nvalid - tc * ZT);
        if (nv <= 0) continue;
        const int streams = ZT / nv;
        const int stream = tid / nv;
        const bool active = stream < streams;
        const int tile = active ? list_sh[tid - stream * nv] : 0;
        const int a0 = 4 * (tile / tcols), b0 = 2 * (tile % tcols);
        float acc[8][10];
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int q = 0; q < 10; ++q) acc[e][q] = 0.f;
        float2 g[ZIT][5];
        float w1[ZIT], wr[ZIT], wi[ZIT];
        bool on[ZIT];
        auto load = [&](int c0) {
#pragma unroll
            for (int j = 0; j < ZIT; ++j) {
                const int idx = tid + j * ZT;
                const int v = idx / nb, a = idx - v * nb;
                on[j] = v < chunk && c0 + v < sg.y && (a >= nbd ? a - nbd : a) >= ks;
                if (!on[j]) continue;
                const float* R = Q.rec + 4 * (size_t)Q.order[sg.x + c0 + v];
                const float2* RG = reinterpret_cast<const float2*>(R + 8 + 6 * nb) + a - col0;
                w1[j] = R[3]; wr[j] = R[4]; wi[j] = R[5];
                g[j][0] = RG[(n - sh + M + 1) * ncol];      // G[n-1]
                g[j][1] = RG[(-n - sh + M + 1) * ncol];     // G[-n-1]
                g[j][2] = RG[(n + sh + M + 1) * ncol];      // G[n+1]
                g[j][3] = RG[(-n + sh + M + 1) * ncol];     // G[-n+1]
                g[j][4] = RG[(gst + n) * ncol];             // W[n]
            }
        };
        auto store = [&](float4* T) {
#pragma unroll
            for (int j = 0; j < ZIT; ++j) {
                if (!on[j]) continue;
                const int idx = tid + j * ZT;
                const float2 gm1 = g[j][0], gmm1 = g[j][1], gp1 = g[j][2], gmp1 = g[j][3], w = g[j][4];
                T[idx] = make_float4(wr[j] * gm1.x - wi[j] * gm1.y, wr[j] * gm1.y + wi[j] * gm1.x,     // A0
                                     wr[j] * gp1.x + wi[j] * gp1.y, wr[j] * gp1.y - wi[j] * gp1.x);    // A1
                T[comp + idx] = make_float4(wr[j] * gmp1.x + wi[j] * gmp1.y,                           // A3
                                            wi[j] * gmp1.x - wr[j] * gmp1.y, w1[j] * w.x, w1[j] * w.y);
                T[2 * comp + idx] = make_float4(gmm1.x, gmm1.y, gmp1.x, gmp1.y);                       // B0, B1
                T[3 * comp + idx] = make_float4(gp1.x, -gp1.y, w.x, -w.y);                             // B2, BW
            }
        };
        load(0);
        store(zsh);
        __syncthreads();
        for (int c0 = 0, buf = 0; c0 < sg.y; c0 += chunk, buf ^= 1) {
            const bool more = c0 + chunk < sg.y;
            if (more) load(c0 + chunk);
            const float4* T = zsh + buf * 4 * comp;
            const int nvr = min(chunk, sg.y - c0);
            if (active) {
                for (int v = stream; v < nvr; v += streams) {
                    const float4* pa = T + v * nb + a0;
                    const float4* pb = T + 2 * comp + v * nb + b0;
                    const float4 b01[2] = {pb[0], pb[1]}, b2w[2] = {pb[comp], pb[comp + 1]};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 a01 = pa[i], a3w = pa[comp + i];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            float* f = acc[2 * i + j];
                            const float4 x = b01[j], y = b2w[j];
                            f[0] = fmaf(-a01.y, x.y, fmaf(a01.x, x.x, f[0]));
                            f[1] = fmaf(a01.y, x.x, fmaf(a01.x, x.y, f[1]));
                            f[2] = fmaf(-a01.w, x.w, fmaf(a01.z, x.z, f[2]));
                            f[3] = fmaf(a01.w, x.z, fmaf(a01.z, x.w, f[3]));
                            f[4] = fmaf(-a01.y, y.y, fmaf(a01.x, y.x, f[4]));
                            f[5] = fmaf(a01.y, y.x, fmaf(a01.x, y.y, f[5]));
                            f[6] = fmaf(-a3w.y, x.y, fmaf(a3w.x, x.x, f[6]));
                            f[7] = fmaf(a3w.y, x.x, fmaf(a3w.x, x.y, f[7]));
                            f[8] = fmaf(-a3w.w, y.w, fmaf(a3w.z, y.z, f[8]));
                            f[9] = fmaf(a3w.w, y.z, fmaf(a3w.z, y.w, f[9]));
                        }
                    }
                }
            }
            if (more) store(zsh + (buf ^ 1) * 4 * comp);
            __syncthreads();
        }
        if (!active) continue;
        double* part = Q.part + (size_t)n * 80 * ntile + tile;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int a = a0 + (e >> 1), b = b0 + (e & 1);
            const int m = min(a >= nbd ? a - nbd : a, b >= nbd ? b - nbd : b);
            if (a >= nb || b >= nb || m < ks || m >= mk) continue;
#pragma unroll
            for (int q = 0; q < 10; ++q)
                atomicAdd(part + (size_t)(q * 8 + e) * ntile, (double)acc[e][q]);
        }
    }
}

}  // namespace

size_t zeta_part_doubles(int nb, int M)
{ return (size_t)(M + 1) * 80 * (((nb + 3) >> 2) * ((nb + 1) >> 1)); }

long long zeta_segments(long long nrec, int nb, int nbd)
{ return nrec / (nb > MANY_BINS ? RUN_MANY : SEG_MIN) + (long long)nbd * (nbd + 1) + 1; }

int launch_zeta(const ZParams& Q, int nsm, cudaStream_t st)
{
    const int chunk = std::min(64, std::max(1, ZIT * ZT / Q.nbins));
    const size_t sm = sizeof(float4) * 8 * (size_t)(chunk * Q.nbins + ZPAD);
    TC_TRY(allow_smem(k_mp_zeta, sm));
    TC_CU(cudaMemsetAsync(Q.count, 0, sizeof(int) * (size_t)Q.nbd * (Q.nbd + 1), st));
    const int blocks = (int)std::min<long long>(4LL * nsm, (Q.nrec + 255) / 256);
    count_launch();
    k_zrows<<<blocks, 256, 0, st>>>(Q, false);
    count_launch();
    k_zrows_segments<<<1, 1024, 0, st>>>(Q);
    count_launch();
    k_zrows<<<blocks, 256, 0, st>>>(Q, true);
    count_launch();
    k_mp_zeta<<<2 * nsm, ZT, sm, st>>>(Q);
    TC_CU(cudaGetLastError());
    return 0;
}

}  // namespace tc
