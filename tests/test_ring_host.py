"""Which copies of a ring a warp that gives up waits for (tilus_b200/csrc/ring.cuh), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "ring.cuh"
extern "C" int last_wait(int slot, int issued, int slots) {  // -1: none
  const b200q::RingLaps laps = b200q::ring_laps(issued, slots);
  return b200q::ring_used(laps, slot) ? (int)b200q::ring_parity(laps, slot) : -1;
}
"""


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    base = tmp_path_factory.mktemp("ring")
    (base / "ring.cpp").write_text(SOURCE)
    out = str(base / "ring.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "tilus_b200", "csrc"),
                           str(base / "ring.cpp"), "-o", out])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("slots", range(1, 9))
def test_a_wait_passes_when_its_copy_has_landed_and_not_before(ring, slots):
    """An mbarrier's wait for a parity passes unless the phase under way has it.  Every number of items asked for, every number of
    them landed that the ring allows (an item is asked for when the one `slots` ahead of it has landed)."""
    for issued in range(1, 5 * slots + 2):
        for landed in range(max(0, issued - slots), issued + 1):
            for slot in range(slots):
                uses = [i for i in range(issued) if i % slots == slot]
                parity = ring.last_wait(slot, issued, slots)
                assert (parity < 0) == (not uses)
                if uses:
                    under_way = sum(1 for i in uses if i < landed)  # phases of the slot's barrier that have ended
                    assert (parity != under_way % 2) == (uses[-1] < landed), (issued, landed, slot)
