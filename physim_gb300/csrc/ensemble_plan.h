// ensemble_plan.h -- how an ensemble cuts a member's j range into one-pair units
// (host arithmetic only).
#pragma once

#include <algorithm>

namespace pg {

// Most j chunks a member of n bodies is split into (sizes the partial sums).  An
// empty member (a slot that waits for its next job) counts as one chunk.
inline int most_splits(int n)
{
    return std::max(1, std::max((n + 4095) / 4096, std::min(8, (n + 255) / 256)));
}

// A member's j range in tiles of `block` bodies: chunk_tiles to a chunk, `splits`
// chunks, at most most_splits(n).
struct MemberCut {
    int n_jtiles, chunk_tiles, splits;
};

inline MemberCut cut_member(int n, int block, int chunk)
{
    const int most = most_splits(n);
    MemberCut c;
    c.n_jtiles = (n + block - 1) / block;
    chunk = std::max(chunk, (n + most - 1) / most);
    c.chunk_tiles = std::max(1, (chunk + block - 1) / block);
    c.splits = std::max(1, (c.n_jtiles + c.chunk_tiles - 1) / c.chunk_tiles);
    return c;
}

}  // namespace pg
