"""The Tensor surface's paged attention of steps with prompts in them: on the tensor core, with split probabilities.  The oracle
is the CPU restatement; what a call leaves to the general kernel is compared with the f32 call on the same values, which that
kernel serves whole."""
import numpy as np
import pytest
import torch

from oracle import oracle
from singe_b200 import kernel_sys as ks, ops, workloads
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

PAGE = 16


def step(rng, new, every, heads, kv_heads, dim, spare=3):
    counts = [-(-n // PAGE) for n in every]
    pool = sum(counts) + spare
    paging = {"query_offsets": np.concatenate([[0], np.cumsum(new)]), "page_offsets": np.concatenate([[0], np.cumsum(counts)]),
              "pages": rng.permutation(pool)[: sum(counts)],
              "last_page_lengths": np.asarray([(n - 1) % PAGE + 1 if n else 0 for n in every])}
    q = workloads.normal_bf16(rng, (sum(new), heads, dim))
    return q, workloads.normal_bf16(rng, (pool, PAGE, kv_heads, dim)), workloads.normal_bf16(rng, (pool, PAGE, kv_heads, dim)), paging


def run_step(q, kc, vc, paging, kind=torch.bfloat16, index=np.int64, **options):
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    tensors = [t.to(kind) if isinstance(t, torch.Tensor) else dev(t, kind) for t in (q, kc, vc)]
    out, lse = ops.paged_attention(*tensors, *(dev(paging[name].astype(index)) for name in
                                               ("query_offsets", "page_offsets", "pages", "last_page_lengths")),
                                   scale=tensors[0].shape[2] ** -0.5, status=status, **options)
    torch.cuda.synchronize()
    return host(out), host(lse), int(status.item())


def assert_rounded(out, ref, what):
    """``out`` is ``ref`` rounded to bf16 (half a unit: 2^-8), up to what probabilities of 2^-17 relative error and f32 sums of
    values below 6 leave."""
    assert (np.abs(out - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-4).all(), f"{what}: {np.abs(out - ref).max()}"


def assert_log_sums(lse, ref):
    """Of the largest score's size, some 20 here, or of the log sum where that is larger: eight steps of the tensor core, which drops
    what lies below its accumulator's last bit (2^-23 each), and a few roundings of either side's exponentials and sums."""
    worst = np.abs(lse - ref) / np.maximum(20.0, np.abs(ref))
    assert worst.size == 0 or worst.max() < 20 * 2.0 ** -24, worst.max()


NEW = [1, 300, 0, 70, 1, 33, 1, 256, 2]
EVERY = [517, 300, 40, 900, 16, 20, 1, 640, 0]     # more keys than new tokens, as many, fewer, none


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (4, 4, 128), (8, 1, 64), (6, 2, 64), (32, 2, 128), (4, 2, 128)])
@pytest.mark.parametrize("causal,window,index", [(True, 0, np.int64), (False, 0, np.int32), (True, 100, np.int64), (True, 1, np.int32),
                                                 (True, 5000, np.int64)])
def test_steps_with_prompts(heads, kv_heads, dim, causal, window, index):
    rng = np.random.default_rng(heads + dim + window)
    q, kc, vc, paging = step(rng, NEW, EVERY, heads, kv_heads, dim)
    out, lse, status = run_step(q, kc, vc, paging, index=index, causal=causal, window=window)
    code, ref, ref_lse = oracle.attend_paged_f32(q, kc, vc, *paging.values(), scale=dim ** -0.5, causal=causal, window=window)
    assert code == oracle.OK and status == 0 and ops.take_device_error() == 0
    assert_rounded(out, ref, "out")
    assert (np.isneginf(lse) == np.isneginf(ref_lse)).all()
    seen = np.isfinite(ref_lse)
    assert_log_sums(lse[seen], ref_lse[seen])


def test_rows_of_no_sequence_are_left_alone():
    rng = np.random.default_rng(3)
    q, kc, vc, paging = step(rng, [40, 3, 20], [40, 80, 33], 8, 2, 128)
    paging["query_offsets"] = np.asarray([5, 45, 45, 60])
    out, lse, status = run_step(q, kc, vc, paging)
    ref, ref_lse, _ = run_step(q, kc, vc, paging, torch.float32)
    assert status == 0 and not out[:5].any() and not out[60:].any() and np.isneginf(lse[:5]).all()
    assert_rounded(out, ref, "out")
    assert_log_sums(lse[5:60], ref_lse[5:60])


def same_as_general(q, kc, vc, paging):
    """The bf16 call against the f32 call on the same values."""
    out, lse, status = run_step(q, kc, vc, paging)
    ref, ref_lse, ref_status = run_step(q, kc, vc, paging, torch.float32)
    assert status == ref_status
    for mine, other in ((out, ref), (lse, ref_lse)):
        assert (np.isnan(mine) == np.isnan(other)).all() and (np.isinf(mine) == np.isinf(other)).all()
    fine = np.isfinite(ref)
    assert_rounded(out[fine], ref[fine], "out")
    fine = np.isfinite(ref_lse)
    assert_log_sums(lse[fine], ref_lse[fine])
    return status


@pytest.mark.parametrize("fault", ["page", "last", "page_offsets", "query_offsets", "backwards"])
def test_paging_out_of_range_leaves_the_other_sequences_whole(fault):
    rng = np.random.default_rng(11)
    q, kc, vc, paging = step(rng, NEW, EVERY, 8, 2, 128)
    if fault == "page":
        paging["pages"][paging["page_offsets"][3] + 20] = kc.shape[0]    # rows before that page's keys are still computed
    elif fault == "last":
        paging["last_page_lengths"][1] = PAGE + 1
    elif fault == "page_offsets":
        paging["page_offsets"][-1] += 1
    elif fault == "query_offsets":
        paging["query_offsets"][-1] += 1
    else:
        paging["query_offsets"][4] -= 100
    assert same_as_general(q, kc, vc, paging) == 1
    q, kc, vc, paging = step(rng, NEW, EVERY, 8, 2, 128)                 # and the next call is served as ever
    assert same_as_general(q, kc, vc, paging) == 0


@pytest.mark.parametrize("what", ["hidden values", "hidden keys", "seen value", "infinite value", "unused slots", "jump", "all hidden low"])
def test_values_the_tensor_core_cannot_carry(what):
    rng = np.random.default_rng(13)
    q, kc, vc, paging = step(rng, [200, 1, 30], [260, 300, 30], 8, 2, 128)
    at = lambda sequence, key: (paging["pages"][paging["page_offsets"][sequence] + key // PAGE], key % PAGE)
    if what == "hidden values":
        vc[at(0, 200)] = np.nan           # seen from row 140 on
    elif what == "hidden keys":
        kc[at(0, 200)] = np.inf
    elif what == "seen value":
        vc[at(1, 7)] = np.nan
    elif what == "infinite value":
        vc[at(1, 7)] = np.inf
    elif what == "unused slots":
        vc[at(2, 30)] = np.nan
        vc[at(0, 260)] = np.inf
    elif what == "jump":
        kc[at(0, 150)] = 60.0 * np.sign(q[150, 0])   # scores that outgrow the first key tile's by far more than 2^64
    else:
        q[:, 0] = 2.0 ** 100
        kc[at(0, 0)] = -2.0 ** 100        # a score of minus infinity
    same_as_general(q, kc, vc, paging)


def on_gpu(q, kc, vc, paging):
    names = ("query_offsets", "page_offsets", "pages", "last_page_lengths")
    return [dev(t, torch.bfloat16) for t in (q, kc, vc)] + [dev(paging[name].astype(np.int64)) for name in names]


def test_a_faulty_call_leaves_no_trace():
    # 2000 tokens on 32 heads: what a later call would look up again is a fifth of its time
    rng = np.random.default_rng(23)
    new = [500] * 4 + [1] * 28
    q, kc, vc, paging = step(rng, new, [n + int(c) for n, c in zip(new, rng.integers(0, 3000, len(new)))], 32, 8, 128)
    tensors = on_gpu(q, kc, vc, paging)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call = lambda: ops.paged_attention(*tensors, status=status)

    def time():
        events = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = []
        for _ in range(10):
            events[0].record()
            for _ in range(10):
                call()
            events[1].record()
            events[1].synchronize()
            best.append(events[0].elapsed_time(events[1]))
        return min(best)

    call()
    before, (out, lse) = time(), call()
    assert status.item() == 0
    page = tensors[5][40].item()
    tensors[5][40] = kc.shape[0]
    call()
    assert status.item() == 1
    tensors[5][40] = page
    kc_word = tensors[1][page, 0].clone()
    tensors[1][page, 0] = float("nan")         # and one with values that are not finite
    assert call()[0].isnan().any()
    tensors[1][page, 0] = kc_word
    again, lse_again = call()
    assert torch.equal(again, out) and torch.equal(lse_again, lse)
    assert time() < 1.08 * before               # runs of one build differ by 1 - 2 %


def test_captured_steps_and_streams_of_their_own():
    rng = np.random.default_rng(29)
    steps = [step(rng, NEW, EVERY, 8, 2, 128) for _ in range(2)]
    tensors = [on_gpu(*s) for s in steps]
    statuses = [torch.zeros(1, dtype=torch.int32, device="cuda") for _ in steps]
    expected = [ops.paged_attention(*t, status=s) for t, s in zip(tensors, statuses)]
    pages = tensors[1][5]
    page, bad = pages[-1].item(), steps[1][1].shape[0] + 5
    pages[-1] = bad
    refused = ops.paged_attention(*tensors[1], status=statuses[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = ops.paged_attention(*tensors[1], status=statuses[1])
    for id, wanted in ((page, expected[1]), (bad, refused), (page, expected[1])):
        pages[-1] = id
        graph.replay()
        assert all(torch.equal(*pair) for pair in zip(captured, wanted))
    pages[-1] = bad
    streams = [torch.cuda.Stream() for _ in steps]
    torch.cuda.synchronize()
    found = [[], []]
    for _ in range(20):                         # the one is refused while the other is not, and they overlap
        for own, stream, t, s in zip(found, streams, tensors, statuses):
            with torch.cuda.stream(stream):
                own.append(ops.paged_attention(*t, status=s))
    torch.cuda.synchronize()
    assert statuses[0].item() == 0 and statuses[1].item() == 1
    for own, wanted in zip(found, (expected[0], refused)):
        assert all(torch.equal(*pair) for result in own for pair in zip(result, wanted))


def test_a_cache_without_pages():
    tensors = [torch.zeros((5, 4, 128), dtype=torch.bfloat16, device="cuda")] * 3
    out, lse = torch.full_like(tensors[0], 7.0), torch.full((5, 4), 7.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    paging = [torch.tensor(v, device="cuda") for v in ([0, 3, 3, 5], [0, 0, 0, 0], [0], [0, 0, 0])]
    code = ks.lib().singe_paged_attention_bf16(int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), lse.data_ptr(),
                                               *(t.data_ptr() for t in tensors + paging), 8, 5, 4, 2, 128, PAGE, 0, 3, 0, 0.1, 1, 0,
                                               status.data_ptr())
    torch.cuda.synchronize()
    assert code == ks.OK and status.item() == 0 and not out.any() and bool(lse.isneginf().all())
