// mrmg_pending.cuh -- places in the list of undecided positions (arm edges).
// Compiles as host C++ too, so the counting is tested there near its limits.
#pragma once

#include "mrmg_exact.cuh"

namespace mrmg {

// The list's count is an int: a call has up to 2^31 edges of up to 2^24
// positions, any of which may be undecided, so the count stops where the list
// does.  A longer scratch block is used up to here.
constexpr long long kMaxPending = (1ll << 31) - (1ll << 26);

MRMG_HD long long pend_room(long long cap) { return cap < kMaxPending ? cap : kMaxPending; }

// The caller's place in a list of `cap` entries, or -1: full.  A warp that finds
// the list full says so (lose) and counts no more, nor does a warp that reads it
// (lost): the count passes pend_room(cap) by at most one per warp of the launch.
template <class Count>
MRMG_HD int pend_claim(Count& c, long long cap) {
  if (c.lost()) return -1;
  const int slot = c.add();
  if (slot < pend_room(cap)) return slot;
  c.lose();
  return -1;
}

// Entries that were written, of the count a launch has left
MRMG_HD int pend_listed(int count, long long cap) { return count < pend_room(cap) ? count : (int)pend_room(cap); }

}  // namespace mrmg
