"""The Tensor surface's paged attention where a query tile stands alone and its key tiles alternate between two places, and
where more (sequence, row pair) entries come than are put in order.  Bounds as in the tests of steps with prompts."""
import numpy as np
import pytest

from oracle import oracle
from singe_b200 import ops
from tests.test_gpu_tensor_prompts import assert_log_sums, assert_rounded, run_step, same_as_general, step

import torch

pytestmark = pytest.mark.gpu

TILE = 128


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (8, 1, 64), (4, 4, 128)])
@pytest.mark.parametrize("causal,window", [(True, 0), (False, 0), (True, 130), (True, 400)])
def test_lone_query_tiles(heads, kv_heads, dim, causal, window):
    # one to nine key tiles, ending one key before, at and after a tile's edge; pairs of tiles and empty sequences between
    rng = np.random.default_rng(heads + dim + window)
    new = [1, 2, 1, 3, 300, 1, 1, 30, 1, 0, 1, 2]
    every = [TILE, TILE + 1, 2 * TILE - 1, 2 * TILE, 700, 2 * TILE + 1, 3 * TILE, 3 * TILE + 5, 5 * TILE + 1, 9, 0, 9 * TILE - 3]
    q, kc, vc, paging = step(rng, new, every, heads, kv_heads, dim)
    out, lse, status = run_step(q, kc, vc, paging, causal=causal, window=window)
    code, ref, ref_lse = oracle.attend_paged_f32(q, kc, vc, *paging.values(), scale=dim ** -0.5, causal=causal, window=window)
    assert code == oracle.OK and status == 0 and ops.take_device_error() == 0
    assert_rounded(out, ref, "out")
    assert (np.isneginf(lse) == np.isneginf(ref_lse)).all()
    seen = np.isfinite(ref_lse)
    assert_log_sums(lse[seen], ref_lse[seen])


@pytest.mark.parametrize("what", ["second place weightless", "first place weightless", "second place minus infinity", "jump in second",
                                  "infinite value in second", "hidden value behind the last"])
def test_values_in_either_place(what):
    rng = np.random.default_rng(17)
    q, kc, vc, paging = step(rng, [1, 2], [2 * TILE, 3 * TILE - 8], 4, 1, 128)
    at = lambda sequence, key: (paging["pages"][paging["page_offsets"][sequence] + key // 16], key % 16)
    q[:] = np.abs(q)
    keys = lambda first, last, value: [kc.__setitem__(at(0, key), value) for key in range(first, last)]
    if what == "second place weightless":
        keys(TILE, 2 * TILE, -40.0)
    elif what == "first place weightless":
        keys(0, TILE, -40.0)
    elif what == "second place minus infinity":
        q[0] = 2.0 ** 100
        keys(TILE, 2 * TILE, -2.0 ** 100)
        keys(0, TILE, 0.0)
    elif what == "jump in second":
        kc[at(1, TILE + 5)] = 60.0
    elif what == "infinite value in second":
        vc[at(0, TILE + 1)] = np.inf
    else:
        vc[at(1, 3 * TILE - 8)] = np.nan
    same_as_general(q, kc, vc, paging)


def test_more_entries_than_are_ordered():
    rng = np.random.default_rng(19)
    new = [1] * 1020 + [1500]
    every = [int(n) for n in rng.integers(1, 300, size=1020)] + [1600]
    q, kc, vc, paging = step(rng, new, every, 2, 2, 64)
    out, lse, status = run_step(q, kc, vc, paging)
    ref, ref_lse, _ = run_step(q, kc, vc, paging, torch.float32)
    assert status == 0
    assert_rounded(out, ref, "out")
    assert_log_sums(lse, ref_lse)
