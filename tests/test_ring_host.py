"""Which copies of a ring a warp that gives up waits for (tilus_b200/csrc/ring.cuh), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "ring.cuh"
extern "C" int slot(int item, int slots) { return b200q::ring_slot(item, slots); }
extern "C" int parity(int item, int slots) { return (int)b200q::ring_parity(item, slots); }
extern "C" int oldest(int issued, int slots) { return b200q::ring_oldest(issued, slots); }
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
            under_way = [sum(1 for i in range(landed) if i % slots == s) for s in range(slots)]  # phases ended, per slot
            waits = range(ring.oldest(issued, slots), issued)
            assert set(range(landed, issued)) <= set(waits)
            assert sorted(ring.slot(i, slots) for i in waits) == sorted({ring.slot(i, slots) for i in range(issued)})
            for i in waits:
                passes = ring.parity(i, slots) != under_way[ring.slot(i, slots)] % 2
                assert passes == (i < landed), (issued, landed, i)
