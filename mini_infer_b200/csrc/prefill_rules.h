// Rules of the tcgen05 prompt attention that are plain arithmetic, in standard C++, so that they can be checked without a
// device.
#pragma once

#include <cstdint>

namespace mi {
namespace pt {

constexpr int BQ = 128;            // queries per tile (MMA M)
constexpr int SMS = 148;
// query tiles per block: two, but one where the queries of two would leave no room for rings
constexpr int query_tiles(int dk) { return dk > 192 ? 1 : 2; }

// Which query tiles share a block (and its key tiles):
//   kSingle      one alone, where the tiles of all heads and requests find an SM each (or two do not fit): a chain by
//                itself takes 0.80 us a key tile, two beside each other 1.05 us
//   kApart       the last but i and the first but i, where the pairs find an SM each and all earlier keys are seen: no
//                block has two long ones (2,048 queries of 16 heads, 128 blocks: 36 us, 45 us with neighbours)
//   kNeighbours  2 i and 2 i + 1, whose keys are nearly the same, so that both chains run to the end (8,192 queries of 16
//                heads: 263 us, 353 us apart)
// The lengths are on the device: tiles and pairs are bounded by `longest` rows for every request and by `total` rows with one
// tile (or pair) begun for every request.
enum QueryTiles : int { kSingle = 0, kApart = 1, kNeighbours = 2 };
constexpr int64_t least_of(int64_t a, int64_t b) { return a < b ? a : b; }
constexpr int64_t parts_at_most(int64_t longest, int64_t total, int requests, int64_t rows) {
    return least_of((longest + rows - 1) / rows * requests, total / rows + requests);
}
constexpr QueryTiles query_order(int64_t longest, int64_t total, int heads, int requests, int dk, bool bounded) {
    if (query_tiles(dk) == 1 || parts_at_most(longest, total, requests, BQ) * heads <= SMS) return kSingle;
    return !bounded && parts_at_most(longest, total, requests, 2 * BQ) * heads <= SMS ? kApart : kNeighbours;
}

// Whether a softmax warp waits for O += P V of key tile j - 1 of n before it hands over P of tile j (`rescale`: it changes
// O first).  A wait on a parity tells only neighbouring phases apart, and a parity that is two phases behind never
// comes, so every such wait stands BEFORE the hand-over: product j cannot complete without this warp, and S of tile j was
// issued after product j - 2, which leaves the barrier in phase j - 1 or j.  At the last tile the wait is there even
// without a rescale: behind the hand-over the last two products may complete before a warp looks, and only what it saw
// before tells phase n - 2 from phase n.  (That product was issued a tile ago, so this seldom waits.)
constexpr bool follows_product(int j, int n, bool rescale) { return j > 0 && (rescale || j == n - 1); }

}  // namespace pt
}  // namespace mi
