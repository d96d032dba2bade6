"""What the host decides about the even form of paged decode, and what the fold may read."""
import ctypes

import pytest

from singe_b200 import kernel_sys as ks


@pytest.mark.parametrize("slots", [2, 5, 149, 300])
def test_fold_stays_inside_its_scratch(slots):
    # whatever stands in a list's entry: slots - 1 of them hold partials, the last one is the list
    inside = ks.lib()._ZN5singe15even_row_insideEiii
    inside.argtypes, inside.restype = [ctypes.c_int] * 3, ctypes.c_bool
    edges = sorted({0, 1, 2, slots - 3, slots - 2, slots - 1, slots, 256, 257, 2 ** 31 - 1, -1, -2, -2 ** 31, 2 ** 31 - slots})
    for segments in edges:
        for slot in edges:
            assert inside(segments, slot, slots) == (0 < segments <= 256 and slot >= 0 and slot + segments <= slots - 1)
