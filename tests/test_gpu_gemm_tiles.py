"""Linear layers at the edges of their tilings: pairs of SMs from 129 rows on, one row tile with K split or not below.

The bound is that of f32 sums of exact bf16 products in any order, K * 2^-23 * sum |x| |w|, and half an ulp of bf16 (2^-8 of
the value, and of the bound's) where the result is rounded to it.
"""
import pytest
import torch

from singe_b200 import kernel_sys as ks
from singe_b200 import ops

pytestmark = pytest.mark.gpu


def _inputs(m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn((m, k), generator=gen, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=gen, device="cuda") * 0.05).to(torch.bfloat16)
    exact = x.double() @ w.double().T
    bound = k * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    return x, w, exact, bound


def _check(got, exact, bound, what):
    error = (got.double() - exact).abs()
    limit = bound if got.dtype == torch.float32 else bound + 2.0 ** -8 * (exact.abs() + bound)
    assert bool((error <= limit).all()), f"{what}: {float((error - limit).max())} beyond the bound"


def _linear(out, x, w, activation):
    code = ks.lib().singe_linear_bf16(int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), x.data_ptr(), w.data_ptr(),
                                      x.shape[0], w.shape[0], x.shape[1], x.stride(0), w.stride(0), out.stride(0), activation, 0)
    assert code == ks.OK


@pytest.mark.parametrize("width", [0, 64, 128, 192, 224, 256])
@pytest.mark.parametrize("m,n,k", [(129, 64, 64), (255, 258, 72), (257, 1000, 520), (385, 2050, 136), (3000, 9736, 64)])
def test_pairs_of_sms(m, n, k, width):
    # one row past a row tile, one column pair past a column tile, K tails, several tiles for a pair, a pair with half a tile
    x, w, exact, bound = _inputs(m, n, k)
    lib = ks.lib()
    aligned = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    odd = torch.full((m, n + 3), float("nan"), dtype=torch.bfloat16, device="cuda")
    wide = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    gated = torch.full((m, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
    gated_odd = torch.full((m, n // 2 + 1), float("nan"), dtype=torch.bfloat16, device="cuda")
    halves = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    squared = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    chain = torch.empty((m, n // 2), dtype=torch.bfloat16, device="cuda")
    assert lib.singe_matmul_set_tuning(width, 1 if width else 0) == ks.OK
    try:
        _linear(aligned, x, w, 0)
        _linear(odd[:, :n], x, w, 0)
        ops.matmul_bf16(wide, x, w, ops.MatmulConfig.row_major_transposed_rhs(m, n, k))
        _linear(gated, x, w, 1)
        _linear(gated_odd[:, : n // 2], x, w, 1)
        _linear(halves, x, torch.cat([w[0::2], w[1::2]]).contiguous(), 0)
        _linear(squared, x, w, 2)
    finally:
        assert lib.singe_matmul_set_tuning(0, 0) == ks.OK
    assert lib.singe_silu_mul_bf16(int(torch.cuda.current_stream().cuda_stream), chain.data_ptr(), halves.data_ptr(),
                                   halves.data_ptr() + n // 2 * 2, halves.stride(0), m, n // 2) == ks.OK
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    _check(wide, exact, bound, "f32")
    _check(aligned, exact, bound, "bf16")
    assert torch.equal(odd[:, :n], aligned) and bool(odd[:, n:].isnan().all())
    assert torch.equal(gated, chain) and torch.equal(gated_odd[:, : n // 2], gated)
    assert bool(gated_odd[:, n // 2:].isnan().all())
    assert torch.equal(squared, wide.clamp_min(0).square().to(torch.bfloat16))


@pytest.mark.parametrize("m,n,k", [(129, 128, 72), (300, 1000, 136), (1000, 9736, 64)])
def test_pairs_of_sms_with_a_right_operand_of_k_rows(m, n, k):
    x, w, exact, bound = _inputs(m, n, k)
    right = w.T.contiguous()
    out = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    ops.matmul_bf16(out, x, right, ops.MatmulConfig(m, n, k, x.stride(0), right.stride(0), n, False, False))
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    _check(out, exact, bound, "f32")


@pytest.mark.parametrize("m", [1, 64, 65, 96, 128])
@pytest.mark.parametrize("n,k", [(64, 2048), (768, 4096), (2048, 8192), (2304, 2048), (4096, 768), (6144, 2048), (8200, 1024),
                                 (9480, 520), (10240, 264)])
def test_one_row_tile(m, n, k):
    # where the rule turns: 8, 4, 2 and no splits, tiles of 64 and 128 columns, K too short to split
    x, w, exact, bound = _inputs(m, n, k)
    out = ops.linear(x, w)
    gated_odd = torch.full((m, n // 2 + 1), float("nan"), dtype=torch.bfloat16, device="cuda")
    gated = torch.full((m, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
    _linear(gated_odd[:, : n // 2], x, w, 1)
    _linear(gated, x, w, 1)
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    _check(out, exact, bound, "bf16")
    assert torch.equal(gated_odd[:, : n // 2], gated) and bool(gated_odd[:, n // 2:].isnan().all())


@pytest.mark.parametrize("m,n,k,parts", [(64, 6144, 4096, 2), (128, 6144, 4096, 2), (64, 4096, 4096, 4), (128, 4096, 4096, 4),
                                         (1, 8192, 2048, 2), (128, 8192, 2048, 2), (1, 4608, 2048, 4), (100, 2304, 2048, 4),
                                         (16, 768, 4096, 8), (96, 1400, 4096, 8), (64, 8200, 1000, 2), (33, 4100, 1544, 4),
                                         (128, 9600, 4096, 1)])
def test_partial_sums_of_one_row_tile(m, n, k, parts):
    # K is cut for the sums by N and K alone, however the work is shared out: the bits are those of one CTA for every partial sum
    x, w, exact, bound = _inputs(m, n, k)
    got = []
    for splits in (0, parts):
        assert ks.lib().singe_matmul_set_splits(splits) == ks.OK
        try:
            out = torch.full((m, n), float("nan"), device="cuda")
            ops.matmul_bf16(out, x, w, ops.MatmulConfig.row_major_transposed_rhs(m, n, k))
            got.append(out)
        finally:
            assert ks.lib().singe_matmul_set_splits(0) == ks.OK
    torch.cuda.synchronize()
    assert ops.take_device_error() == 0
    _check(got[0], exact, bound, "f32")
    assert torch.equal(*got)
