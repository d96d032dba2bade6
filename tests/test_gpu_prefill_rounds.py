"""Prompt attention of more items than a CTA decodes ahead, and outputs that whole-sector stores do not reach."""
import numpy as np
import pytest
import torch

from oracle import oracle
from singe_b200 import ops, workloads
from tests.gpu_util import assert_close_bf16, assert_close_f32, dev, host

pytestmark = pytest.mark.gpu


# 64 items are decoded ahead: one more a CTA, and a few; an output on a 32-byte boundary and half a sector behind one
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("sequences", [3, 310])
def test_many_items_and_shifted_outputs(head_dim, shift, sequences):
    heads, kv_heads = 32, 8
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lens = np.asarray([5 + (7 * i) % 19 for i in range(sequences)], dtype=np.int32)
    assert (sequences * heads > 64 * sms) == (sequences == 310)
    offsets = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int32)
    total, rng, scale = int(lens.sum()), np.random.default_rng(sequences + shift), head_dim ** -0.5
    q = workloads.normal_bf16(rng, (total, heads, head_dim))
    k, v = (workloads.normal_bf16(rng, (total, kv_heads, head_dim)) for _ in range(2))
    room = torch.full((total * heads * head_dim + 32,), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = room[shift: shift + total * heads * head_dim].view(total, heads, head_dim)
    assert out.data_ptr() % 32 == 2 * shift
    lse = torch.full((total, heads), float("nan"), device="cuda")
    ops.ragged_kv_prefill_attention(out, lse, *[dev(x, torch.bfloat16) for x in (q, k, v)], dev(lens), dev(lens), dev(offsets),
                                    ops.RaggedKvPrefillAttentionConfig(sequences, total, total, heads, kv_heads, head_dim, True, scale))
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    expect, expect_lse = oracle.ragged_kv_prefill_attention_f32(q, k, v, lens, lens, offsets, batch=sequences, total_query_tokens=total,
                                                                heads=heads, kv_heads=kv_heads, head_dim=head_dim, causal=True, scale=scale)
    assert_close_bf16(host(out), expect, "out")
    assert_close_f32(host(lse), expect_lse, "lse", 2e-4)   # log2 and exp2 approximations: 2^-22 of |score| below 16, a few of them
    assert room[:shift].isnan().all() and room[shift + total * heads * head_dim:].isnan().all()


# the most items for which every CTA has one only, and one pair of rows more
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("more", [0, 1])
def test_one_item_for_every_sm(head_dim, more):
    heads, kv_heads, sequences = 4, 2, 20
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    total = (sms // heads - sequences + more) * 256 + 3
    assert ((total // 256 + sequences) * heads <= sms) == (more == 0)
    lens = np.full(sequences, 130, dtype=np.int32)
    lens[3], lens[7] = 1, total - 18 * 130 - 1
    offsets = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int32)
    rng, scale = np.random.default_rng(more), head_dim ** -0.5
    q = workloads.normal_bf16(rng, (total, heads, head_dim))
    k, v = (workloads.normal_bf16(rng, (total, kv_heads, head_dim)) for _ in range(2))
    out = torch.full((total, heads, head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    lse = torch.full((total, heads), float("nan"), device="cuda")
    ops.ragged_kv_prefill_attention(out, lse, *[dev(x, torch.bfloat16) for x in (q, k, v)], dev(lens), dev(lens), dev(offsets),
                                    ops.RaggedKvPrefillAttentionConfig(sequences, total, total, heads, kv_heads, head_dim, True, scale))
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    expect, expect_lse = oracle.ragged_kv_prefill_attention_f32(q, k, v, lens, lens, offsets, batch=sequences, total_query_tokens=total,
                                                                heads=heads, kv_heads=kv_heads, head_dim=head_dim, causal=True, scale=scale)
    assert_close_bf16(host(out), expect, "out")
    assert_close_f32(host(lse), expect_lse, "lse", 2e-4)
