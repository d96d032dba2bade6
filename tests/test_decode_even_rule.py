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


@pytest.mark.parametrize("kv_heads,head_dim,batch,bound,pays", [
    # few rows; ragged batches that lost, and the same from where they no longer do; rows of one piece each
    (8, 128, 4, 1600, True), (8, 128, 1, 6000, False), (8, 128, 6, 1030, True), (8, 128, 64, 128, False), (8, 128, 64, 160, True),
    (8, 128, 32, 4096, True), (8, 64, 4, 4224, True), (8, 64, 6, 2800, True), (8, 64, 7, 2800, False), (8, 64, 20, 1024, False),
    (8, 64, 15, 1911, False), (8, 64, 22, 876, True), (8, 64, 20, 2500, True), (8, 64, 64, 400, True), (4, 64, 24, 2128, False),
    (4, 64, 43, 2200, False), (4, 64, 44, 2200, True), (4, 64, 32, 4480, True), (4, 128, 4, 3200, True), (4, 128, 5, 2600, False),
    (4, 128, 8, 2048, True), (4, 128, 20, 900, False), (4, 128, 20, 1632, True), (4, 128, 64, 512, True),
    (8, 64, 73, 512, True), (8, 64, 74, 512, False), (8, 64, 81, 528, True), (8, 128, 73, 200, True), (8, 128, 74, 200, False),
    (8, 128, 74, 272, True), (4, 128, 148, 512, False), (4, 128, 147, 512, True)])
def test_drop_in_calls_take_the_even_form_where_ragged_batches_do_not_lose(kv_heads, head_dim, batch, bound, pays):
    rule = ks.lib()._ZN5singe22paged_decode_even_paysEmmmm
    rule.argtypes, rule.restype = [ctypes.c_size_t] * 4, ctypes.c_bool
    assert rule(batch, kv_heads, head_dim, bound) == pays
    if bound != 512:      # (whole pages count, but for the line at 512 keys)
        assert rule(batch, kv_heads, head_dim, bound // 16 * 16 - 15) == rule(batch, kv_heads, head_dim, bound // 16 * 16)


def test_positions_of_the_even_form_stay_below_2_31():
    splits = lambda bound: ks.lib().singe_paged_kv_decode_even_splits(1, 32, 8, 128, bound, 16)
    assert splits(2 ** 31 - 32) > 0 and splits(2 ** 31 - 16) > 0 and splits(2 ** 31) == 0 and splits(2 ** 34) == 0
