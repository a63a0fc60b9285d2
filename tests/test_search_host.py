"""The room that an active search without a cap asks for: one call where its
first guess is enough, a second of exactly the size found where it is not, and
never more than 2 MB for the guess, however long the list (no GPU)."""
import ctypes

import numpy as np
import pytest

from glint_pipeline_gb300 import DeviceBench


class Library:
    """glint_active_search with `found` entries for any list"""

    def __init__(self, found):
        self.found, self.rooms = found, []

    def glint_active_search(self, h, pids, npids, out, cap, n):
        self.rooms.append(cap)
        written = min(cap, self.found)
        if written:
            ctypes.memset(out, 7, 32 * written)
        n._obj.value = self.found
        return 0


@pytest.mark.parametrize("npids,found,rooms", [
    (1, 4096, [4096]), (1, 4097, [4096, 4097]), (1000, 5, [32000]),
    (10_000_000, 5, [1 << 16]), (10_000_000, 1 << 20, [1 << 16, 1 << 20]),
])
def test_room_without_a_cap(npids, found, rooms):
    g = DeviceBench.__new__(DeviceBench)
    g.lib, g.h = Library(found), None
    got = g.active_search(np.zeros(npids, np.uint32))
    assert g.lib.rooms == rooms and len(got) == found
    assert np.all(got.view(np.uint8) == 7)


def test_room_with_a_cap():
    g = DeviceBench.__new__(DeviceBench)
    g.lib, g.h = Library(50), None
    assert len(g.active_search(np.zeros(3, np.uint32), cap=20)) == 20
    assert len(g.active_search(np.zeros(3, np.uint32), cap=0)) == 0
    assert g.lib.rooms == [20, 0]
