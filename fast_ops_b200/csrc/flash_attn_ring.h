// The order in which a warp that issues matmuls takes the entries of a ring of K and V tiles.
// Plain C++, so that the same code runs in the kernel and in a model of the ring's barriers on the CPU.
//
// Entry 2 j is the K tile of key tile j in the CTA's order, entry 2 j + 1 its V tile; entry e is the
// (e / kStages)-th use of slot e % kStages, and its load completes phase e / kStages of the slot's
// "full" barrier.  A slot is loaded again once both issuing warps have released it.
//
// A barrier is waited on by the parity of a phase: the wait for phase f returns as soon as the
// barrier is not in phase f - 1 + 2 n, so a warp that has not seen phase f - 1 end may be let
// through one load early, and loads do not complete in the order they were requested in.  Hence the
// rule that this walk keeps: a warp waits for every entry, in order within a slot, also for those it
// only passes over.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define FO_RING_FN __device__ __forceinline__
#else
#define FO_RING_FN inline
#endif

namespace fo {

// The walk of a warp whose query tile takes the steps `first` (0 or 1) to `end` - 1, two per key tile, on
// the key tiles j0 to j1 - 1 of the n that the ring carries (the others belong to the CTA's other query
// tile).
//   ops.wait(slot, parity)      blocks until that phase of the slot's "full" barrier is complete
//   ops.ready(slot, parity)     the same without blocking
//   ops.release(slot)           this warp's readers of the slot have all been issued
//   ops.scores(t, slot)         issues the scores of step t, one of the first two, whose K tile is in `slot`
//   ops.step(t, v_slot, k_slot) issues P V of step t and the scores of step t + 2 if there is one
template <int kStages, class Ops>
FO_RING_FN void walk_kv_ring(int j0, int j1, int n, int first, int end, const Ops& ops) {
  auto slot = [](int e) { return e % kStages; };
  auto parity = [](int e) { return static_cast<uint32_t>((e / kStages) & 1); };
  auto pass_over = [&](int e, int e_end) {
    for (; e < e_end; ++e) {
      ops.wait(slot(e), parity(e));
      ops.release(slot(e));
    }
  };
  pass_over(0, 2 * j0);
  ops.wait(slot(2 * j0), parity(2 * j0));
  ops.scores(first, slot(2 * j0));
  if (first == 0 && end > 1) ops.scores(1, slot(2 * j0));
  ops.release(slot(2 * j0));
  if (first == 1 && end > 2) {
    ops.wait(slot(2 * j0 + 2), parity(2 * j0 + 2));
    ops.scores(2, slot(2 * j0 + 2));
  }
  bool ready = false;  // looked at one step ahead, waited for only if that look failed
  for (int t = first; t < end; ++t) {
    const int j = (t >> 1) + j0;
    const int v = 2 * j + 1, k = v + 1;  // V of this step's key tile, K of the next
    const bool k_next = j + 1 < j1;
    if (((t & 1) == 0 || t == first) && !ready) {
      ops.wait(slot(v), parity(v));
      if (k_next) ops.wait(slot(k), parity(k));
    }
    ready = false;
    ops.step(t, slot(v), slot(k));
    if ((t & 1) == 1 || t + 1 == end) {
      ops.release(slot(v));
      if (k_next) ops.release(slot(k));
      if (t + 1 < end) ready = ops.ready(slot(v + 2), parity(v + 2)) && (!(j + 2 < j1) || ops.ready(slot(k + 2), parity(k + 2)));
    }
  }
  pass_over(2 * j1, 2 * n);
}

}  // namespace fo
