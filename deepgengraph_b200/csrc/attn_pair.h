// How the two warps that share the rows of a query tile agree (attn_fwd_split.cuh).  Plain C++ over three operations, so that the
// order of the steps can be run on the host under many interleavings:
//   vote(x)      barrier of both warps; true in both if x was true anywhere
//   put(x)/get() write the own exchange word / read the partner's
//
// A word is rewritten only after a barrier that its reader joins later than its read:
//   * in a block, after the block's vote;
//   * at the end of a tile, after the wait for the tile's last P V: that product needs the P of both warps, and a warp delivers its
//     P after it has read its partner's word.
//
// A step is one vote, and a second one where the first came out true.  The second vote says whether a bounded wait of either warp ran
// out; then both leave.  It is the barrier's own answer, so both get the same one (a flag in shared memory could be raised by the
// partner's next step before it is read, and the partner would then wait in that step alone).
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define B200_PAIR_FN __host__ __device__ __forceinline__
#else
#define B200_PAIR_FN inline
#endif

namespace b200 {

enum class PairStep { kKeep, kMoved, kLeave };

// One block.  `ok`: its S has arrived; `moves`: the reference maximum of one of this warp's rows has to move.  After kMoved, `m_blk`
// is the maximum over both halves of the row.
template <class Pair>
B200_PAIR_FN PairStep pair_block(const Pair& w, bool ok, bool moves, float& m_blk) {
  if (!w.vote(!ok || moves)) return PairStep::kKeep;
  w.put(m_blk);
  if (w.vote(!ok)) return PairStep::kLeave;
  m_blk = fmaxf(m_blk, w.get());
  return PairStep::kMoved;
}

// A wait ran out between two steps: takes part in the partner's next step.
template <class Pair>
B200_PAIR_FN void pair_leave(const Pair& w) {
  w.vote(true);
  w.vote(true);
}

// End of a tile: `l` becomes the sum over both halves of the row.  `wait_o` waits for the tile's last P V.
template <class Pair, class WaitO>
B200_PAIR_FN bool pair_total(const Pair& w, WaitO wait_o, float& l) {
  const bool ok = wait_o();
  if (ok) w.put(l);
  if (w.vote(!ok)) {
    w.vote(!ok);
    return false;
  }
  l += w.get();
  return true;
}

// No more tiles: the partner may have failed where this warp did not.
template <class Pair>
B200_PAIR_FN void pair_finish(const Pair& w) {
  if (w.vote(false)) w.vote(false);
}

}  // namespace b200
