// A warp's ring of shared-memory slots: item i is the (i / slots)-th use of slot i % slots, one phase of the slot's mbarrier each.  Plain
// integer C++, so that a test checks it on the host.
#pragma once
#include "decode.cuh"

namespace b200q {

B200Q_HD constexpr int ring_slot(int item, int slots) { return item % slots; }
// what a wait for the item's copy names (a phase two uses back has the same parity, but ended before this one began)
B200Q_HD constexpr uint32_t ring_parity(int item, int slots) { return (uint32_t)(item / slots) & 1u; }
// the oldest of the `issued` items whose copy may still be on its way: a slot is asked for again when its last copy has landed
B200Q_HD constexpr int ring_oldest(int issued, int slots) { return issued > slots ? issued - slots : 0; }

}  // namespace b200q
