"""Dense f32 attention in tiles against the CPU restatement."""
import numpy as np
import pytest
import torch

from oracle import oracle
from singe_b200 import kernel_sys as ks, ops
from tests.gpu_util import assert_close_f32, dev, host

pytestmark = pytest.mark.gpu


def attend(q, k, v, scale, causal, window=0, softcap=0.0, sinks=None):
    b, h, l, d = q.shape
    out = torch.full((b, h, l, d), float("nan"), device="cuda")
    code = ks.lib().singe_attend_f32(int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), q.data_ptr(), k.data_ptr(),
                                     v.data_ptr(), b, h, k.shape[1], l, k.shape[2], d, scale, int(causal), window, softcap,
                                     None if sinks is None else sinks.data_ptr())
    torch.cuda.synchronize()
    assert code == ks.OK
    return out


# few rows and the first past a tile's edge, one team of threads and two, heads that fill neither width, more queries than keys
@pytest.mark.parametrize("b,h,g,l,s,d", [(1, 2, 1, 16, 16, 64), (1, 3, 3, 33, 200, 20), (2, 4, 2, 65, 65, 64), (1, 2, 2, 130, 63, 128),
                                         (1, 6, 3, 97, 129, 72), (4, 16, 4, 300, 300, 64), (3, 26, 13, 257, 321, 96)])
@pytest.mark.parametrize("causal,window,softcap,with_sinks", [(True, 0, 0.0, False), (False, 0, 0.0, True), (True, 21, 1.5, True),
                                                              (False, 70, 0.0, False)])
def test_dense_f32_tiles(b, h, g, l, s, d, causal, window, softcap, with_sinks):
    rng = np.random.default_rng(b * 1000 + l)
    q, k, v = (rng.standard_normal(shape, dtype=np.float32) for shape in ((b, h, l, d), (b, g, s, d), (b, g, s, d)))
    sinks = rng.standard_normal(h).astype(np.float32) if with_sinks else None
    out = attend(dev(q), dev(k), dev(v), d ** -0.5, causal, window, softcap, dev(sinks) if with_sinks else None)
    wide = lambda x: np.repeat(x, h // g, axis=1)
    ref = oracle.attend_options_f32(q, wide(k), wide(v), scale=d ** -0.5, causal=causal, window=window, softcap=softcap, sinks=sinks)
    # f32 sums over at most s + d terms of values below 6: 2^-24 * 450 * 6 = 1.6e-4 at worst, the root of that many in practice
    assert_close_f32(host(out), ref, "dense f32", 2e-5)


def test_dense_f32_lse_and_what_hidden_keys_hold():
    rng = np.random.default_rng(5)
    b, l, h, g, d = 2, 150, 4, 2, 64
    q, k, v = (torch.from_numpy(rng.standard_normal((b, l, n, d), dtype=np.float32)).cuda() for n in (h, g, g))
    run = lambda: (torch.empty_like(q), torch.empty((b, h, l), device="cuda"))
    out, lse = run()
    call = lambda out, lse: ops.fmha_prefill_lse(out, lse, q, k, v, batch=b, query_len=l, key_len=l, heads=h, kv_heads=g, head_dim=d,
                                                 scale=0.125, causal=True)
    call(out, lse)
    scores = torch.einsum("blhd,bshd->bhls", q.double(), k.double().repeat_interleave(h // g, 2)) * 0.125
    scores.masked_fill_(torch.ones(l, l, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    assert (lse.double() - scores.logsumexp(3)).abs().max() < 1e-5
    k[:, 100], v[:, 101], v[:, 102] = float("nan"), float("inf"), float("nan")
    again, lse_again = run()
    call(again, lse_again)
    assert torch.equal(again[:, :100], out[:, :100]) and torch.equal(lse_again[:, :, :100], lse[:, :, :100])
    assert again[:, 102:].isnan().any(-1).all()


@pytest.mark.parametrize("l", [15, 16, 40, 300])       # one warp per row, and tiles
@pytest.mark.parametrize("b,d", [(1, 64), (1, 128), (120, 64), (120, 128)])   # two and four teams of threads, two and one
def test_dense_f32_sinks_that_are_not_finite(l, b, d):
    rng = np.random.default_rng(l)
    s, window, h = l - 12, 5, 4                        # the last seven rows see no key
    q, k, v = (dev(rng.standard_normal((b, h, n, d), dtype=np.float32)) for n in (l, s, s))
    sinks = torch.tensor([float("-inf"), 0.5, float("inf"), float("nan")], device="cuda")
    out = attend(q, k, v, 0.125, False, window, 0.0, sinks)
    assert not out[:, :, s + window - 1:].any()        # zero for every sink: nothing is weighed, whatever the sum is
    assert torch.equal(out[:, 0], attend(q, k, v, 0.125, False, window)[:, 0])
    assert out[:, :2].isfinite().all() and out[:, 2:, : s + window - 1].isnan().all()


@pytest.mark.parametrize("d", [16, 32, 48, 64, 72, 96, 128])
@pytest.mark.parametrize("l", [16, 24, 40, 100])
@pytest.mark.parametrize("causal", [True, False])
def test_dense_f32_error_is_no_larger_than_one_warp_per_rows(d, l, causal):
    # Inputs four bytes off go by one warp per row.  The same values, 128 heads: the two mean errors are known to about 1 %
    # (1024 row means of errors of some 0.5 each, correlated along a row), so two of those are allowed.
    gen = torch.Generator(device="cuda").manual_seed(d * 1000 + l)
    q, k, v = (torch.randn((16, 8, l, d), generator=gen, device="cuda") for _ in range(3))
    shifted = torch.empty(q.numel() + 1, device="cuda")[1:].view(q.shape).copy_(q)
    scores = q.double() @ k.double().transpose(-1, -2) * d ** -0.5
    if causal:
        scores.masked_fill_(torch.ones(l, l, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    exact = torch.softmax(scores, -1) @ v.double()
    tiles, warps = ((attend(x, k, v, d ** -0.5, causal).double() - exact).norm() for x in (q, shifted))
    assert tiles <= 1.02 * warps
