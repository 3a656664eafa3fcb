// Turn order of the two softmax groups of the attention forward kernel.
//
// Group 0 owns the first query tile of an item, group 1 the second.  They take turns on the unit that evaluates the
// exponentials: 0, 1, 0, 1, ...  A barrier per group counts its turns, and a waiter sees no more of a count than its parity,
// so the rule has to keep each group within one turn of what the other has waited for:
//   * only blocks that both tiles have take a turn (min of the two block counts of an item; a causal item's second tile has
//     one block more, a last tile may be missing).  The count is therefore the same for both groups at all times;
//   * group 0 waits before turn k for the other's turn k - 1, in every item, group 1 for the other's turn k.
// Group 0 cannot start turn k + 1 before group 1 has finished turn k, and group 1 cannot finish turn k before group 0 has:
// at a wait for turn k the awaited count is k or k + 1, which its parity tells apart, however late a warp looks.
// (With the unmatched block counted as well, and no wait at the first block of an item, a group could finish two turns
// before a slow warp of the other looked at the first, and both then waited for good.)
//
// Plain C++, so that the CPU tests can walk every interleaving of it.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FT_TURNS_FN __host__ __device__ __forceinline__
#else
#define FT_TURNS_FN inline
#endif

namespace ftk {

struct AttnTurns {
  uint32_t before;      // turns of the items before this one
  int n;                // turns of this item
  FT_TURNS_FN AttnTurns() : before(0), n(0) {}
  // next item: key blocks of its two tiles
  FT_TURNS_FN void item(int blocks0, int blocks1) {
    before += (uint32_t)n;
    n = blocks0 < blocks1 ? blocks0 : blocks1;
  }
  // block j is a turn: its exponentials end with an arrival on the group's barrier
  FT_TURNS_FN bool takes(int j) const { return j < n; }
  // group t waits before block j; `parity`: phase of the other group's barrier
  FT_TURNS_FN bool waits(int t, int j, uint32_t& parity) const {
    const uint32_t k = before + (uint32_t)j;
    parity = (t == 0 ? k - 1u : k) & 1u;
    return j < n && (t != 0 || k > 0);
  }
};

}  // namespace ftk
