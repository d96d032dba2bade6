"""Dense f32 attention whose row tiles are shared by two CTAs, against 64-bit sums."""
import pytest
import torch

from singe_b200 import kernel_sys as ks

pytestmark = pytest.mark.gpu


# one key past the first tiles of both CTAs' teams, a CTA without keys of its own, a last step for one CTA only, partial row tiles,
# more queries than keys; then the most tiles the rule takes (74 of any kind, 118 of long causal walks) and one head more
@pytest.mark.parametrize("h,g,l,s", [(2, 1, 33, 129), (3, 3, 16, 193), (4, 2, 200, 257), (2, 2, 300, 140), (1, 1, 500, 500), (8, 4, 288, 320),
                                     (37, 37, 64, 130), (38, 19, 64, 130), (9, 9, 401, 401), (10, 5, 400, 400)])
@pytest.mark.parametrize("d", [20, 64, 128])
@pytest.mark.parametrize("causal,window,with_sinks", [(True, 0, False), (False, 0, True), (True, 150, True), (False, 131, False)])
def test_shared_row_tiles(h, g, l, s, d, causal, window, with_sinks):
    gen = torch.Generator(device="cuda").manual_seed(l + d)
    q, k, v = (torch.randn(1, n, m, d, device="cuda", generator=gen) for n, m in ((h, l), (g, s), (g, s)))
    sinks = torch.randn(h, device="cuda", generator=gen) if with_sinks else None
    out = torch.full_like(q, float("nan"))
    code = ks.lib().singe_attend_f32(int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), q.data_ptr(), k.data_ptr(),
                                     v.data_ptr(), 1, h, g, l, s, d, d ** -0.5, int(causal), window, 0.0,
                                     None if sinks is None else sinks.data_ptr())
    assert code == ks.OK
    wide = lambda x: x.repeat_interleave(h // g, 1).double()
    scores = q.double() @ wide(k).transpose(-1, -2) * d ** -0.5
    rows = torch.arange(l, device="cuda")[:, None]
    keys = torch.arange(s, device="cuda")[None, :]
    hidden = torch.zeros(l, s, dtype=torch.bool, device="cuda")
    if causal:
        hidden |= keys > rows
    if window:
        hidden |= keys + window <= rows      # (rows past the keys and the window see none)
    scores.masked_fill_(hidden, float("-inf"))
    if with_sinks:
        scores = torch.cat([scores, sinks.double()[None, :, None, None].expand(1, h, l, 1)], -1)
    expect = torch.nan_to_num(torch.softmax(scores, -1))[..., :s] @ wide(v)
    # f32 sums over at most s + d terms of values below 6: 2^-24 * 630 * 6 = 2.3e-4 at worst, the root of that many in practice
    assert (out.double() - expect).abs().max() < 2e-5
