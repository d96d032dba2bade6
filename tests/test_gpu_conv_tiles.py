"""Prompts' attention inputs, tiles of eight rows held in shared memory, against the same rows one at a time."""
import numpy as np
import pytest
import torch

from singe_b200.layer_ops import Ops

pytestmark = pytest.mark.gpu


def check_tiles(heads, kv_heads, taps, dim=128, vdim=128, pairs=32):
    ops, page_size = Ops("bfloat16"), 16
    lengths = [4001, 1, 743]
    tokens = sum(lengths)
    assert tokens >= 4 * torch.cuda.get_device_properties(0).multi_processor_count * 8 and tokens % 8 == 1
    key_at, value_at = heads * dim, (heads + kv_heads) * dim
    span, pages = value_at + kv_heads * vdim, tokens // page_size + 1
    gen = torch.Generator(device="cuda").manual_seed(heads)
    normal = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).bfloat16()
    projected, bias, weight, norms = normal(tokens, span), normal(span), normal(taps, span), (normal(heads * dim), normal(kv_heads * dim))
    frequencies = torch.logspace(0, -4, pairs, dtype=torch.float64, device="cuda")
    i32 = lambda x: torch.as_tensor(np.asarray(x, dtype=np.int32)).cuda()
    i64 = lambda x: torch.as_tensor(np.asarray(x, dtype=np.int64)).cuda()
    first = np.cumsum([0] + lengths)[:-1]
    context, place = [3, 0, 1], np.arange(tokens)
    kept = normal(len(lengths), max(taps - 1, 1), span)[:, :taps - 1].contiguous()

    def run(portions):
        query = torch.zeros((tokens, heads * dim), dtype=torch.bfloat16, device="cuda")
        caches = [torch.zeros((pages, page_size, kv_heads * size), dtype=torch.bfloat16, device="cuda") for size in (dim, vdim)]
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        for begin, end in portions:    # (a portion's rows are all new tokens of a call that starts with the whole prompt's first row)
            n = end - begin
            at = np.arange(begin, end)
            sequence_of = np.searchsorted(first, at, side="right") - 1
            ops.call("singe_conv_attention_inputs_bf16", int(torch.cuda.current_stream().cuda_stream), query[begin:end], query.stride(0),
                     *caches, None, None, projected[begin:end], projected.stride(0), bias, weight, kept.clone(), norms[0], norms[1],
                     frequencies, pairs, 1.0, i64(at), i32(sequence_of), i32(first - begin), i32(lengths), i32(context),
                     i64(place[begin:end] // page_size), i64(place[begin:end] % page_size), None, None, 0, n, len(lengths), taps, heads,
                     kv_heads, dim, vdim, dim, vdim, key_at, value_at, span, pages, page_size, 1e-5, status)
        assert int(status.item()) == 0
        return [query] + caches

    whole = run([(0, tokens)])
    few = run([(begin, min(begin + 1000, tokens)) for begin in range(0, tokens, 1000)])
    assert all(torch.equal(a, b) for a, b in zip(whole, few)) and whole[0].float().abs().sum() > 0


# rows of 192, 384, 640 and 1024 threads (24 to 136 KB of shared memory); a last tile of one row; a sequence that begins inside a tile
@pytest.mark.parametrize("heads,kv_heads,taps", [(8, 2, 4), (16, 4, 4), (24, 8, 1), (48, 8, 3)])
def test_tiles_equal_rows_one_at_a_time(heads, kv_heads, taps):
    check_tiles(heads, kv_heads, taps)


# 48 KB to the byte behind the kernel's own arrays, from rows of 352, 384 and 320 threads
@pytest.mark.parametrize("heads,kv_heads,taps,dim,vdim,pairs", [(16, 4, 4, 128, 64, 64), (16, 4, 2, 128, 128, 0), (6, 2, 4, 256, 256, 128)])
def test_tiles_of_48_kilobytes(heads, kv_heads, taps, dim, vdim, pairs):
    span = (heads + kv_heads) * dim + kv_heads * vdim
    assert 8 * (span // 8 * 16 + pairs * 8) == 48 * 1024
    check_tiles(heads, kv_heads, taps, dim, vdim, pairs)
