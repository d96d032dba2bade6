"""The step's arrays against a restatement that places one token at a time."""
import itertools
import random
import warnings

import numpy as np
import pytest
import torch

from singe_b200.decoder import PageTable, PageTableError, token_array


def one_by_one(table, tokens, padding):
    """What a step of ``tokens`` holds, from the table before it and the pages it hands out."""
    free, rows = list(table.free), []
    padded = max(i for i, t in enumerate(tokens) if len(t) > 0)
    for row, t in enumerate(tokens):
        held, length = list(table.pages[row]), table.lengths[row]
        for place in (table._unseen(row) if len(t) else []):
            held[place] = table.pool
        for token in t:
            if length // table.page_size == len(held):
                held.append(free.pop())
            rows.append((token, length, held[length // table.page_size], length % table.page_size, row))
            length += 1
        if len(t) == 0:
            rows.append((0, min(length, table.capacity - 1), table.pool, 0, row))
        for position in range(length, length + padding) if row == padded else ():
            rows.append((0, min(position, table.capacity - 1), table.pool, position % table.page_size, row))
    return [list(column) for column in zip(*rows)]


@pytest.mark.parametrize("page,window,chunks", [(1, 0, ()), (3, 0, ()), (4, 5, ()), (2, 0, (4,)), (16, 3, (8,))])
def test_steps_of_any_shape(page, window, chunks):
    rng = random.Random(page + window)
    for _ in range(60):
        sequences, capacity = rng.randint(1, 5), rng.randint(1, 50)
        table = PageTable.create_shared(sequences, capacity, page, sequences * (capacity + page), window, chunks).with_padding(9)
        for _ in range(6):
            tokens = [[rng.randint(0, 99) for _ in range(rng.choice((0, 1, 1, 2, rng.randint(0, 20))))] for _ in range(sequences)]
            padding = rng.choice((0, 0, 1, 9))
            refused = all(not t for t in tokens) or any(n + len(t) > capacity for n, t in zip(table.lengths, tokens))
            before = ([list(p) for p in table.pages], list(table.lengths), list(table.free))
            if refused:
                with pytest.raises(PageTableError):
                    table.step_padded(tokens, table.step_tokens(tokens) + padding)
                assert before == (table.pages, table.lengths, table.free)
                continue
            # pages given back are handed out again within the same step: compare where none are
            given_back = any(table._unseen(row) for row, t in enumerate(tokens) if t)
            expected = one_by_one(table, tokens, padding)
            step = table.step_padded(tokens, table.step_tokens(tokens) + padding)
            got = [step.tokens, step.positions, step.write_pages, step.write_slots, step.sequence_ids]
            for index, (mine, wanted) in enumerate(zip(got, expected)):
                if index != 2 or not given_back:
                    assert mine.dtype == np.int64 and mine.tolist() == wanted
            assert step.real_tokens.tolist() == [len(t) for t in tokens]
            assert table.lengths == [n + len(t) for n, t in zip(before[1], tokens)]


def test_token_ids_come_in_any_sequence_of_integers():
    for tokens in ([3, 5], (3, 5), np.asarray([3, 5], dtype=np.int32), [np.int64(3), True + 4], ["3", 5.9]):
        assert token_array(tokens).tolist() == [3, 5] and token_array(tokens).dtype == np.int64
    assert token_array([]).tolist() == []
    with pytest.raises((TypeError, ValueError)):
        token_array([None])


@pytest.mark.parametrize("tokens", [
    (v for v in (3, 1)), iter([7]), map(int, "12"), range(4), (5, 6), {9}, [], "34", ["8"], [True, 2], [1.9, -2.9], [np.int32(3), 4],
    np.asarray([1.5, 2.5]), np.asarray([7], dtype=np.uint64), np.asarray(["6"]), torch.tensor([1, 2]), torch.tensor([2.5]),
    [torch.tensor(4), torch.tensor(5)], [2 ** 62]], ids=lambda tokens: type(tokens).__name__)
def test_what_counts_as_tokens(tokens):
    tokens = tokens if hasattr(tokens, "__len__") else iter(list(tokens))
    first, second = (tokens, tokens) if hasattr(tokens, "__len__") else itertools.tee(tokens)
    array = token_array(first)
    assert array.dtype == np.int64 and array.tolist() == [int(v) for v in second]


@pytest.mark.parametrize("tokens", [
    [float("nan")], np.asarray([float("nan")]), np.asarray([float("inf")]), [float("inf")], np.asarray([2 ** 63], dtype=np.uint64), [2 ** 63],
    [[1, 2]], [None], ["a"], torch.tensor([float("nan")]), np.zeros((2, 2))], ids=repr)
def test_what_is_no_token_is_refused(tokens):
    with pytest.raises((TypeError, ValueError, OverflowError)), warnings.catch_warnings():
        warnings.simplefilter("error")
        token_array(tokens)
