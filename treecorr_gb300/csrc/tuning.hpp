// tuning.hpp -- how many work items a launch of the 2-point path takes, by default and in the
// autotuner's trials (host arithmetic only).
#pragma once

#include <algorithm>
#include <vector>

namespace tc {

// Items per expansion launch: up to 32M, less for small catalogs (level buffers hold 4
// chunks each: 1 GB per level at the largest size).
inline long long expand_chunk(long long npoints)
{
    long long CH = 1LL << 16;
    while (CH < (1LL << 25) && CH < 2 * npoints) CH <<= 1;
    return CH;
}

// The bin_slop rule: the items of a level at which the depth-first walk takes over from the
// expansion, or 0 where it starts from the ngen top-level pairs.  By default 8 per point, 2^17 to
// 2^21 (chunk, if set, up to 2^21).  With few points per top cell a top-level pair is a small subtree
// already (at 32 x 32 points some 4000 evaluations at most), and the walk starts from those.
// per_pair: pairs of points per top-level pair.
inline long long walk_start(long long chunk, long long npoints, long long ngen, double per_pair)
{
    const long long want = chunk > 0 ? std::min(chunk, 1LL << 21)
                                     : std::max(1LL << 17, std::min(1LL << 21, 8 * npoints));
    return ngen < want && (per_pair > 1024. || ngen < 4096) ? want : 0;
}

// The chunks that the autotuner tries besides the default: powers of two down to an eighth of
// it, each of which makes other launches than those before it.
inline std::vector<long long> tune_chunks(bool walk, long long npoints, long long ngen, double per_pair)
{
    std::vector<long long> out;
    const long long first = walk ? walk_start(0, npoints, ngen, per_pair) : expand_chunk(npoints);
    const long long least = std::max(walk ? 1LL << 16 : 1LL << 21, first >> 3);
    long long ch = 1;
    while (2 * ch < first) ch <<= 1;
    for (; ch >= least; ch >>= 1) {
        out.push_back(ch);
        if (walk && walk_start(ch, npoints, ngen, per_pair) == 0) break;     // (so do all smaller ones)
    }
    return out;
}

}  // namespace tc
