// A warp's ring of shared-memory slots: item i is the (i / slots)-th use of slot i % slots, one phase of the slot's mbarrier each.  Plain
// integer C++, so that a test checks it on the host.
#pragma once
#include "decode.cuh"

namespace b200q {

// The uses of a ring behind which `issued` items have been asked for: how many of them belong to the last lap, its parity, and whether
// there was one before.  (Subtractions: divisions by the run-time number of slots, on a path that only a launch that gives up takes, cost the
// kernel that keeps the activations in registers up to 2 % of every other launch.)
struct RingLaps { int last; uint32_t parity; bool earlier; };
B200Q_HD RingLaps ring_laps(int issued, int slots) {
  RingLaps r = {issued, 0u, issued > slots};
  while (r.last > slots) { r.last -= slots; r.parity ^= 1u; }
  return r;
}
// whether a slot has been asked for, and the parity that a wait for its last copy names (the use two laps back has the same
// parity, but has ended)
B200Q_HD bool ring_used(const RingLaps& r, int slot) { return slot < r.last || r.earlier; }
B200Q_HD uint32_t ring_parity(const RingLaps& r, int slot) { return slot < r.last ? r.parity : r.parity ^ 1u; }

}  // namespace b200q
