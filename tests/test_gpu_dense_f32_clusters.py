"""Dense f32 attention against 64-bit sums: row tiles that two CTAs share, and last key tiles."""
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


# a last key tile of 1 to 64 keys, for each form: two and four teams, 64 rows
@pytest.mark.parametrize("last", [1, 31, 32, 33, 63, 64])
@pytest.mark.parametrize("h,before,d", [(80, 64, 64), (80, 320, 64), (80, 128, 128), (200, 128, 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_last_tiles(last, h, before, d, causal):
    l = s = before + last
    gen = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(1, h, m, d, device="cuda", generator=gen) for m in (l, s, s))
    out = torch.full_like(q, float("nan"))
    code = ks.lib().singe_attend_f32(int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), q.data_ptr(), k.data_ptr(),
                                     v.data_ptr(), 1, h, h, l, s, d, d ** -0.5, int(causal), 0, 0.0, None)
    assert code == ks.OK
    scores = q.double() @ k.double().transpose(-1, -2) * d ** -0.5
    if causal:
        scores.masked_fill_(torch.ones(l, s, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    expect = torch.softmax(scores, -1) @ v.double()
    # f32 sums over at most s + d terms of values below 6: 2^-24 * 512 * 6 = 1.8e-4 at worst, the root of that many in practice
    assert (out.double() - expect).abs().max() < 2e-5
