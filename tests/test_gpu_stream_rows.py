"""The step between sublayers of several residual streams: few rows, which one CTA pass holds in registers, and many."""
import numpy as np
import pytest
import torch

from singe_b200.layer_ops import Ops

pytestmark = pytest.mark.gpu


# widths that fill the last warp, leave lanes idle, need a second warp by four columns, and are too wide for the few-row form
@pytest.mark.parametrize("rows", [1, 17, 2 * 148, 2 * 148 + 1])
@pytest.mark.parametrize("width,count", [(2048, 4), (2044, 4), (132, 2), (4, 1), (640, 3), (2052, 4), (256, 5)])
@pytest.mark.parametrize("dtype,parts,store", [("bfloat16", 2, 1), ("float32", 1, 0)])
def test_stream_step(rows, width, count, dtype, parts, store):
    ops, gen = Ops(dtype), torch.Generator(device="cuda").manual_seed(rows * width)
    draw = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    pitch = (width + 7) // 8 * 8
    streams, delta = draw(rows, count, width), draw(rows, pitch + width).to(ops.dtype)
    gains, norm = [draw(width).to(ops.dtype) for _ in range(2)], draw(width).to(ops.dtype)
    mix, out, into = draw(count, count), draw(count), draw(count)
    x, y = streams.double(), delta[:, :width].double()
    unit = lambda t: t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-5)
    if parts == 2:
        y = 0.5 * (unit(y) * gains[0].double() + unit(delta[:, pitch:].double()) * gains[1].double())
    expect = torch.einsum("st,rsw->rtw", mix.double(), x) + out.double()[None, :, None] * y[:, None]
    normed_expect = unit(torch.einsum("t,rtw->rw", into.double(), expect)) * norm.double() * 0.7
    normed, held = torch.full((rows, pitch), float("nan"), dtype=ops.dtype, device="cuda"), streams.clone()
    pair = gains if parts == 2 else (None, None)
    ops.call(f"singe_stream_step_norm_{ops.suffix}", int(torch.cuda.current_stream().cuda_stream), held, delta, delta.stride(0), parts, pitch,
             *pair, 0.5, mix, out, into, store, normed, normed.stride(0), norm, 0.7, rows, count, width, 1e-5)
    # f32 sums of at most 2048 squares and 5 products; a normed value is rounded to the activations' type
    if store:
        assert (held.double() - expect).abs().max() <= 4e-6 * expect.abs().max()
    else:
        assert torch.equal(held, streams)
    error = (normed[:, :width].double() - normed_expect).abs()
    assert (error <= (2.0 ** -8 if dtype == "bfloat16" else 1e-5) * normed_expect.abs() + 1e-5).all()
    assert normed[:, width:].isnan().all()
