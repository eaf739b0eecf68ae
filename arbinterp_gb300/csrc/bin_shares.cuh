// Shares of crowded bins (sorted.cu).  Host and device, no CUDA header: the
// arithmetic can be checked on the CPU over the whole range of row counts.
#pragma once

#include <stdint.h>

namespace arb {

// A staged kernel takes one bin per CTA.  Clouds crowd a few bins, and small
// grids have fewer bins than the GPU has CTAs, so a bin of more than bin_share()
// records is cut.
// About four items for each of ~600 resident CTAs.  Where the bins alone make
// two, only a bin of twice the mean is cut (its tile is staged again for every
// share: cutting 1220-record bins at 512 cost 10 %).  At least 512, and nq / 6 a
// bin at most, for the room of the list of further shares.
constexpr uint32_t bin_share(int64_t nbins, int64_t nq) {
  int64_t s = nq / 2432;
  if (nbins >= 1216 && s < 2 * nq / nbins) s = 2 * nq / nbins;
  if (s < nq / (6 * nbins)) s = nq / (6 * nbins);
  return (uint32_t)(s + 1 > 512 ? s + 1 : 512);
}

// Shares of a bin of n records beyond its first.
constexpr uint32_t bin_more_shares(uint32_t n, uint32_t share) { return n > share ? (n - 1) / share : 0; }

// Share `part` of a bin that begins at record `begin` and ends at `end`: its first
// record and its end.  Record numbers reach 2^32 - 1, so first + share is not
// compared with an end: it can wrap.  Nor is a thread's next record, unless all rows
// are at most STAGED_ROWS (the staged evaluators; above, rows are evaluated one lane
// a record): the adjoint compares distances from the first record instead, which
// keep one register more alive in every loop (spills in the float64 evaluators).
constexpr int64_t STAGED_ROWS = 0xffffffffLL - 1024;
constexpr uint32_t bin_first(uint32_t begin, uint32_t part, uint32_t share) { return begin + part * share; }
constexpr uint32_t bin_end(uint32_t first, uint32_t end, uint32_t share) {
  return end - first < share ? end : first + share;
}

}  // namespace arb
