// Buffers and barriers of the footprint ring of coef3_tma_kernel (coef_tc.cu).
// Host and device, no CUDA header: the hand-offs can be checked on the CPU.
#pragma once

#include <stdint.h>

namespace arb {

// Tile k's footprint lies in buffer k mod BUFS and is read by producer group k
// mod GROUPS.  A wait on a parity tells a phase from its neighbours only, so a
// barrier's phases must all be waited for by one thread group, in order: were
// the "full" barriers one a buffer, two groups would take turns on each, and a
// group that is a tile ahead would take the phase before the other group's for
// its own (with three buffers: group 0 at tile 6 while tile 3 is still on its
// way into the same buffer).  So tiles count up to BUFS * GROUPS of them.  The
// "empty" barriers have one waiter, the loader.
template <int BUFS, int GROUPS>
struct FootprintRing {
  static constexpr int FULL = BUFS * GROUPS;  // "full" barriers
  static constexpr int buffer(int k) { return k % BUFS; }
  static constexpr int full(int k) { return k % FULL; }
  static constexpr uint32_t full_parity(int k) { return (uint32_t)(k / FULL) & 1u; }
  static constexpr uint32_t empty_parity(int k) { return (uint32_t)(k / BUFS) & 1u; }
};

}  // namespace arb
