// Rules of the tcgen05 prompt attention that are plain arithmetic, in standard C++, so that they can be checked without a
// device.
#pragma once

namespace mi {
namespace pt {

// Whether a softmax warp waits for O += P V of key tile j - 1 of n before it hands over P of tile j (`rescale`: it changes
// O first).  A wait on a parity tells only neighbouring phases apart, and a parity that is two phases behind never
// comes, so every such wait stands BEFORE the hand-over: product j cannot complete without this warp, and S of tile j was
// issued after product j - 2, which leaves the barrier in phase j - 1 or j.  At the last tile the wait is there even
// without a rescale: behind the hand-over the last two products may complete before a warp looks, and only what it saw
// before tells phase n - 2 from phase n.  (That product was issued a tile ago, so this seldom waits.)
constexpr bool follows_product(int j, int n, bool rescale) { return j > 0 && (rescale || j == n - 1); }

}  // namespace pt
}  // namespace mi
