// ensemble_plan.h -- how an ensemble cuts a member's j range into one-pair units
// (host arithmetic only).
#pragma once

#include <algorithm>

namespace pg {

// Most j chunks a member of n bodies is split into, by any plan (sizes the partial
// sums).  An empty member (a slot that waits for its next job) counts as one chunk.
constexpr int kMinChunk = 4096;
inline int member_splits(int n, int chunk)
{
    return std::max(1, std::max((n + chunk - 1) / chunk, std::min(8, (n + 255) / 256)));
}
inline int most_splits(int n) { return member_splits(n, kMinChunk); }

// A member's j range in tiles of `block` bodies: chunk_tiles to a chunk, `splits`
// chunks of at most `chunk` (kMinChunk or more) bodies.  Each chunk has a partial
// sum of its own, so the cut follows from the member and the plan alone: a member's
// bits are the same beside any others.
struct MemberCut {
    int n_jtiles, chunk_tiles, splits;
};

inline MemberCut cut_member(int n, int block, int chunk)
{
    const int most = member_splits(n, chunk);
    MemberCut c;
    c.n_jtiles = (n + block - 1) / block;
    c.chunk_tiles = std::max(1, (c.n_jtiles + most - 1) / most);
    c.splits = std::max(1, (c.n_jtiles + c.chunk_tiles - 1) / c.chunk_tiles);
    return c;
}

// Chunks to a unit: as many as leave it at most `even` bodies long, or fewer where the
// member then has as many units.
inline int unit_chunks(const MemberCut &c, int block, long long even)
{
    const long long length = (long long)c.chunk_tiles * block;
    const int most = (int)std::max(1ll, std::min<long long>(c.splits, even / length));
    const int units = (c.splits + most - 1) / most;
    return (c.splits + units - 1) / units;
}

}  // namespace pg
