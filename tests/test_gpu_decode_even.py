"""Paged decode whose CTAs share the cached pages evenly, at the places where runs, segments and folds can go wrong."""
import numpy as np
import pytest
import torch

from oracle import llama_ref, oracle
from singe_b200 import kernel_sys as ks
from singe_b200 import ops, workloads
from singe_b200.layer_ops import Ops
from singe_b200.llama import rotary_tables
from tests.gpu_util import assert_close_bf16, dev, dev_u32, host
from tests.test_gpu_decode import _config, _inputs, _oracle

pytestmark = pytest.mark.gpu

LONG = 65536     # a bound on the lengths that has the even form serve short ones too

# one sequence; runs that end inside, at and before a sequence's last page; empty sequences; more sequences than threads; sequences
# of more segments than the fold has under way at once, with eight, four and one warps for a row
LENGTHS = [[1], [16 * 300], [16 * 148 * 2], [0, 33, 0, 512, 0], [1, 15, 16, 17, 2049, 31, 32, 33, 4097, 100],
           [(37 * i) % 90 for i in range(300)], [5000] + [3] * 40, [3000] + [(211 * i) % 700 for i in range(13)]]


def even_splits(case):
    return ks.lib().singe_paged_kv_decode_even_splits(case.batch, case.heads, case.kv_heads, case.head_dim,
                                                      case.block_table_batch_stride * case.block_size, case.block_size)


@pytest.mark.parametrize("lens", LENGTHS, ids=lambda lens: f"{len(lens)}x{max(lens)}")
@pytest.mark.parametrize("heads,kv_heads,head_dim,dtype", [(32, 8, 128, torch.bfloat16), (16, 8, 64, torch.float16), (16, 4, 128, torch.bfloat16),
                                                           (32, 4, 64, torch.bfloat16), (12, 4, 128, torch.float16)])
def test_even_decode(lens, heads, kv_heads, head_dim, dtype):
    case = workloads.paged_decode_case(seed=3, heads=heads, kv_heads=kv_heads, head_dim=head_dim, lens=lens, max_len=LONG)
    assert even_splits(case) > 0
    q, k, v = _inputs(case, seed=len(lens))
    out = torch.full((case.batch, heads, head_dim), float("nan"), dtype=dtype, device="cuda")
    operands = [dev(x, dtype) for x in (q, k, v)]
    for _ in range(2):      # the workspace is not clean the second time
        ops.paged_kv_decode_attention(out, *operands, dev(case.lens), dev_u32(case.block_table), _config(case))
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    assert_close_bf16(host(out), _oracle(case, q, k, v), f"{len(lens)} sequences")
    assert not host(out)[np.asarray(lens) == 0].any()


def split_grid(case, operands):
    """The call in the split grid with the pieces it chooses for itself."""
    splits = ks.lib().singe_paged_kv_decode_default_splits(case.batch, case.kv_heads, case.block_table_batch_stride * 16, 16)
    attn = torch.empty((case.batch, case.heads, splits, case.head_dim), device="cuda")
    out = torch.empty_like(operands[0])
    ops.paged_kv_decode_splitk_reduce(out, attn, torch.empty(attn.shape[:3], device="cuda"), *operands, splits)
    return out


def test_outputs_at_odd_places_take_the_split_grid_with_its_own_pieces():
    case = workloads.paged_decode_case(seed=12, heads=8, kv_heads=8, head_dim=64, lens=[2500, 30, 700], max_len=LONG)
    q, k, v = _inputs(case, seed=13)
    operands = [dev(x, torch.bfloat16) for x in (q, k, v)] + [dev(case.lens), dev_u32(case.block_table), _config(case)]
    room = torch.empty(q.size + 1, dtype=torch.bfloat16, device="cuda")
    out = room[1:].view(q.shape)
    ops.paged_kv_decode_attention(out, *operands)
    assert even_splits(case) > 0 and out.data_ptr() % 4 == 2
    assert torch.equal(out, split_grid(case, operands))


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 8, 128), (8, 4, 64)])
def test_even_decode_lengths_that_no_table_holds(heads, kv_heads, head_dim):
    # below zero: no keys; beyond the table: all that it holds.  Pages that no sequence holds are not numbers
    bound = 65536 // head_dim * 8
    case = workloads.paged_decode_case(seed=14, heads=heads, kv_heads=kv_heads, head_dim=head_dim, lens=[bound, 40, bound, 300], max_len=bound)
    assert even_splits(case) > 0
    q, k, v = _inputs(case, seed=15)
    held = np.unique(np.concatenate([case.block_table[b, : -(-n // 16)] for b, n in enumerate(case.lens)]))
    spare = np.setdiff1d(np.arange(case.physical_blocks), held)
    assert len(spare) > 0
    k[spare], v[spare] = np.nan, np.inf
    odd = dev(np.asarray([2 ** 31 - 1, -1, bound + 1, -2 ** 31], dtype=np.int32))
    out = torch.full((4, heads, head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    operands = [dev(x, torch.bfloat16) for x in (q, k, v)]
    ops.paged_kv_decode_attention(out, *operands, odd, dev_u32(case.block_table), _config(case))
    case.lens[[1, 3]] = 0
    assert_close_bf16(host(out), _oracle(case, np.nan_to_num(q), np.nan_to_num(k), np.nan_to_num(v)), "odd lengths")
    assert not host(out)[[1, 3]].any() and ops.take_device_error() == 0


@pytest.mark.parametrize("batch", [2048, 2049])
def test_most_sequences_of_the_even_form(batch):
    lens = np.random.default_rng(batch).integers(0, 40, size=batch)
    case = workloads.paged_decode_case(seed=16, heads=32, kv_heads=4, head_dim=128, lens=lens, max_len=1024)
    assert (even_splits(case) > 0) == (batch == 2048)
    q, k, v = _inputs(case, seed=17)
    out = torch.full((batch, 32, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_kv_decode_attention(out, *[dev(x, torch.bfloat16) for x in (q, k, v)], dev(case.lens), dev_u32(case.block_table), _config(case))
    assert_close_bf16(host(out), _oracle(case, q, k, v), f"{batch} sequences")


@pytest.mark.parametrize("heads,kv_heads,head_dim,dtype", [(32, 8, 128, torch.bfloat16), (16, 4, 64, torch.float16)])
def test_even_decode_values_that_are_not_finite(heads, kv_heads, head_dim, dtype):
    # seen values of either infinity and NaN, in a sequence of one segment and in one of many; a finite column beside them
    case = workloads.paged_decode_case(seed=9, heads=heads, kv_heads=kv_heads, head_dim=head_dim, lens=[40, 3000, 17], max_len=LONG)
    assert even_splits(case) > 0
    q, k, v = _inputs(case, seed=10)
    for b in (0, 1):
        for column, value in ((3, np.inf), (4, -np.inf), (5, np.nan)):
            v[case.block_table[b, 1], 2, :, column] = value
    operands = [dev(x, dtype) for x in (q, k, v)] + [dev(case.lens), dev_u32(case.block_table), _config(case)]
    out = torch.empty((case.batch, heads, head_dim), dtype=dtype, device="cuda")
    ops.paged_kv_decode_attention(out, *operands)
    expect = split_grid(case, operands)     # (its weights are one term)
    got, expect = host(out), host(expect)
    assert (expect[:2, :, 3] == np.inf).all() and (expect[:2, :, 4] == -np.inf).all() and np.isnan(expect[:2, :, 5]).all()
    odd = ~np.isfinite(expect)
    assert odd.sum() == 6 * heads and np.array_equal(got[odd], expect[odd], equal_nan=True)
    assert_close_bf16(got[~odd], expect[~odd], "finite columns")


def test_even_decode_reports_page_ids_outside_the_cache():
    case = workloads.paged_decode_case(seed=4, heads=8, kv_heads=4, head_dim=64, lens=[700, 40], max_len=LONG)
    q, k, v = _inputs(case, seed=5)
    table = case.block_table.copy()
    table[0, 20] = case.physical_blocks
    out = torch.empty((2, 8, 64), dtype=torch.bfloat16, device="cuda")
    ops.paged_kv_decode_attention(out, *[dev(x, torch.bfloat16) for x in (q, k, v)], dev(case.lens), dev_u32(table), _config(case))
    assert ops.take_device_error() == ks.STATUS_INDEX_OUT_OF_BOUNDS


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 8, 128), (8, 4, 64)])
@pytest.mark.parametrize("hinted", [False, True])
def test_even_decode_step_adds_its_key(heads, kv_heads, head_dim, hinted):
    # keys including the new one; an idle row; as many sequences as the form wants for a step (over three rows an SM)
    lens = [1, 300, 16, 17, 2049, 0, 513, 33] * (8 if kv_heads == 8 else 14)
    assert len(lens) * kv_heads > 3 * torch.cuda.get_device_properties(0).multi_processor_count
    case = workloads.paged_decode_case(seed=6, heads=heads, kv_heads=kv_heads, head_dim=head_dim, lens=lens, max_len=LONG)
    _, k, v = _inputs(case, seed=7)
    width = (heads + 2 * kv_heads) * head_dim
    qkv = workloads.normal_bf16(np.random.default_rng(8), (case.batch, width))
    positions = np.maximum(np.asarray(lens, dtype=np.int64) - 1, 0)
    pages = np.asarray([case.block_table[b, p // 16] for b, p in enumerate(positions)], dtype=np.int64)
    pages[5::8] = case.physical_blocks - 1        # a page that no sequence holds
    slots = positions % 16
    cos, sin = rotary_tables(head_dim, 500000.0, 4096)
    splits = even_splits(case)
    attn = torch.full((case.batch, heads, splits, head_dim), float("nan"), device="cuda")
    lse = torch.full((case.batch, heads, splits), float("nan"), device="cuda")
    keys, values = dev(k, torch.bfloat16), dev(v, torch.bfloat16)
    out = torch.full((case.batch, heads, head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    device = [dev(qkv, torch.bfloat16), dev(case.lens), dev_u32(case.block_table), dev(cos, torch.bfloat16), dev(sin, torch.bfloat16),
              dev(positions), dev(pages), dev(slots)]
    p = [t.data_ptr() for t in device]
    code = ks.lib().singe_decode_step_attention_bf16(
        int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), attn.data_ptr(), lse.data_ptr(), p[0], width, keys.data_ptr(),
        values.data_ptr(), p[1], p[2], p[3], p[4], p[5], p[6], p[7], 8, case.batch, heads, kv_heads, head_dim, 16,
        case.physical_blocks, case.block_table_batch_stride, splits, 4096, case.scale, ks.HINT_STABLE_PAGING if hinted else 0, None,
        status.data_ptr())
    torch.cuda.synchronize()
    assert code == ks.OK and int(status.item()) == 0 and ops.take_device_error() == 0
    c, s = llama_ref.bf16(cos)[positions], llama_ref.bf16(sin)[positions]
    parts = np.split(qkv.reshape(case.batch, -1, head_dim), [heads, heads + kv_heads], axis=1)
    queries, fresh = llama_ref.rotate(parts[0], c, s), llama_ref.rotate(parts[1], c, s)
    for b, n in enumerate(lens):
        if n > 0:
            k[pages[b], slots[b]], v[pages[b], slots[b]] = fresh[b], parts[2][b]
            assert (host(keys)[pages[b], slots[b]] == fresh[b]).all() and (host(values)[pages[b], slots[b]] == parts[2][b]).all()
    assert_close_bf16(host(out), _oracle(case, queries, k, v), "decode step")


# (the rule leaves short chunks to the split grid, and rows too narrow for the list: both forms are held to the same)
@pytest.mark.parametrize("heads,kv_heads,head_dim,chunk,even", [(16, 4, 128, 512, True), (8, 8, 64, 520, True), (8, 4, 64, 4096, True),
                                                                (8, 8, 64, 100, False), (4, 4, 64, 4096, False)])
def test_even_chunked_decode(heads, kv_heads, head_dim, chunk, even):
    # queries in another order than their sequences, one sequence twice, a query without keys; chunks that begin inside a page
    rng = np.random.default_rng(chunk)
    sequence_of, lens = [2, 0, 1, 1, 3, 0] * 40, [700, 1, 512, 513, 0, 37] * 40
    stride, pool = 64, 256
    table = rng.permutation(pool).reshape(4, stride).astype(np.int32)
    q, k, v = (workloads.normal_bf16(rng, shape) for shape in ((len(lens), heads, head_dim), (pool, 16, kv_heads, head_dim),
                                                                (pool, 16, kv_heads, head_dim)))
    bound = min(chunk + 15, stride * 16)
    splits = ks.lib().singe_paged_kv_decode_even_splits(len(lens), heads, kv_heads, head_dim, bound, 16)
    assert (splits > 0) == even
    splits = splits or 2
    attn = torch.full((len(lens), heads, splits, head_dim), float("nan"), device="cuda")
    lse = torch.full((len(lens), heads, splits), float("nan"), device="cuda")
    out = torch.full((len(lens), heads, head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    i32 = lambda x: dev(np.asarray(x, dtype=np.int32))
    Ops("bfloat16").call("singe_chunked_attention_bf16", int(torch.cuda.current_stream().cuda_stream), out, attn, lse,
                         *[dev(x, torch.bfloat16) for x in (q, k, v)], i32(sequence_of), i32(lens), i32(table), len(lens), heads, kv_heads,
                         head_dim, 16, pool, 4, stride, chunk, splits, head_dim ** -0.5, status)
    assert int(status.item()) == 0
    # the same keys, moved so that each query's chunk begins a page of its own
    first = [(n - 1) // chunk * chunk if n else 0 for n in lens]
    visible = np.asarray([n - f for n, f in zip(lens, first)], dtype=np.int32)
    rows = lambda cache, b: cache[table[b]].reshape(-1, kv_heads, head_dim)
    pages = -(-int(visible.max()) // 16)
    moved = []
    for cache in (k, v):
        parts = np.zeros((len(lens), pages * 16, kv_heads, head_dim), dtype=np.float32)
        for i, (b, f, n) in enumerate(zip(sequence_of, first, lens)):
            parts[i, : n - f] = rows(cache, b)[f:n]
        moved.append(parts.reshape(-1, 16, kv_heads, head_dim))
    expect = oracle.paged_kv_decode_attention_f32(q, *moved, visible, np.arange(len(lens) * pages, dtype=np.uint32).reshape(len(lens), pages),
                                                  batch=len(lens), heads=heads, kv_heads=kv_heads, head_dim=head_dim, block_size=16,
                                                  block_table_batch_stride=pages, scale=head_dim ** -0.5)
    assert_close_bf16(host(out), expect, f"chunks of {chunk}")


def short_problem(seed, dtype=torch.bfloat16):
    """Sequences of at most a piece, which the split grid serves without any scratch; operands and what a lone call gives."""
    lens = np.random.default_rng(seed).integers(1, 513, size=80)
    case = workloads.paged_decode_case(seed=seed, heads=16, kv_heads=8, head_dim=128, lens=lens, max_len=512)
    assert even_splits(case) > 0
    operands = [dev(x, dtype) for x in _inputs(case, seed)] + [dev(case.lens), dev_u32(case.block_table), _config(case)]
    alone = torch.empty_like(operands[0])
    ops.paged_kv_decode_attention(alone, *operands)
    torch.cuda.synchronize()
    assert not torch.equal(alone, split_grid(case, operands))     # (the two forms can be told apart)
    return operands, alone


def test_calls_of_short_sequences_overlap_on_streams():
    problems = [short_problem(seed) for seed in (21, 22)]
    streams = [torch.cuda.Stream() for _ in problems]
    outs = [[torch.empty_like(alone) for _ in range(100)] for _, alone in problems]
    torch.cuda.synchronize()
    for i in range(100):
        for stream, (operands, _), out in zip(streams, problems, outs):
            ops.paged_kv_decode_attention(out[i], *operands, stream=stream)
    torch.cuda.synchronize()
    for (_, alone), out in zip(problems, outs):
        assert all(torch.equal(alone, each) for each in out)


def captured(operands, calls):
    graph, outs = torch.cuda.CUDAGraph(), [torch.empty_like(operands[0]) for _ in range(calls)]
    with torch.cuda.graph(graph):
        for out in outs:
            ops.paged_kv_decode_attention(out, *operands)
    return graph, outs


def test_calls_of_short_sequences_overlap_in_graphs():
    problems = [short_problem(seed) for seed in (23, 24)]
    graphs = [captured(operands, 40) for operands, _ in problems]
    streams = [torch.cuda.Stream() for _ in problems]
    for _ in range(3):
        for _, outs in graphs:
            for out in outs:
                out.zero_()
        torch.cuda.synchronize()
        for stream, (graph, _) in zip(streams, graphs):
            with torch.cuda.stream(stream):
                graph.replay()
        out = torch.empty_like(problems[0][1])
        ops.paged_kv_decode_attention(out, *problems[0][0])       # and a call beside them
        torch.cuda.synchronize()
        assert torch.equal(out, problems[0][1])
        for (_, alone), (_, outs) in zip(problems, graphs):
            assert all(torch.equal(alone, each) for each in outs)


def test_graphs_that_are_gone_give_their_scratch_back():
    operands, alone = short_problem(25)
    for _ in range(150):              # more than there are scratches
        graph, (out,) = captured(operands, 1)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, alone)
        graph.reset()
        torch.cuda.synchronize()


def test_more_graphs_than_scratches():
    operands, alone = short_problem(26)
    kept = [captured(operands, 1) for _ in range(80)]
    for graph, _ in kept:
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(out, alone) for _, (out,) in kept[:8])
    for _, (out,) in kept:            # the last ones in the split grid
        assert_close_bf16(host(out), host(alone), "either form")


def test_a_capture_without_a_call_before_it_is_refused():
    operands, alone = short_problem(27)
    ks.lib().singe_release_workspaces()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(ops.SingeError) as refused:
            ops.paged_kv_decode_attention(torch.empty_like(alone), *operands)
        operands[0].add_(0)
    assert refused.value.code == 12
    ops.paged_kv_decode_attention(alone.clone(), *operands)
    graph, (out,) = captured(operands, 1)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, alone)
