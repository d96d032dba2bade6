"""Norms and rotations of prompts run a warp per row, those of a few rows a CTA per row: one call over many rows gives the bits of
calls over few.  (The few-row kernels are compared with the oracle by their own tests.)"""
import pytest
import torch

from singe_b200 import kernel_sys as ks

pytestmark = pytest.mark.gpu


def _counts():
    """Rows and tokens from which a warp takes one (8 and 12 per SM) with a last CTA that is not full, and too few for that."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 8 * sms + 3, 12 * sms + 5, 3 * sms


def _stream():
    return int(torch.cuda.current_stream().cuda_stream)


def _slices(rows, few):
    return [slice(first, min(first + few, rows)) for first in range(0, rows, few)]


@pytest.mark.parametrize("width", [8, 256, 264, 1024, 1032, 2048, 2056, 4096])
@pytest.mark.parametrize("delta,norm", [(True, True), (False, True), (True, False)])
def test_rms_norm_rows(width, delta, norm):
    rows, _, few = _counts()
    gen = torch.Generator(device="cuda").manual_seed(width)
    normal = lambda *shape: torch.randn(shape, generator=gen, device="cuda").to(torch.bfloat16)
    hidden, change, weight = normal(rows, width), normal(rows, width), normal(width)
    results = []
    for parts in ([slice(0, rows)], _slices(rows, few)):
        h, out = hidden.clone(), torch.zeros_like(hidden)
        for part in parts:
            assert ks.lib().singe_add_rms_norm_bf16(
                _stream(), h[part].data_ptr(), change[part].data_ptr() if delta else None, out[part].data_ptr() if norm else None,
                weight.data_ptr(), h[part].shape[0], width, 1e-5) == ks.OK
        results.append((h, out))
    torch.cuda.synchronize()
    assert all(torch.equal(*pair) for pair in zip(*results))


@pytest.mark.parametrize("kind", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width,padding", [(4, 0), (512, 4), (516, 0), (1028, 0), (1536, 8), (2048, 0), (2052, 0)])
@pytest.mark.parametrize("delta,norm", [(True, True), (False, True), (True, False)])
def test_layer_norm_rows(kind, width, padding, delta, norm):
    rows, _, few = _counts()
    gen = torch.Generator(device="cuda").manual_seed(width)
    residual = torch.randn((rows, width), generator=gen, device="cuda") + 3.0
    change, weight = (torch.randn(shape, generator=gen, device="cuda").to(kind) for shape in ((rows, width + padding), (width,)))
    call = ks.lib().singe_add_layer_norm_bf16 if kind == torch.bfloat16 else ks.lib().singe_add_layer_norm_f32
    results = []
    for parts in ([slice(0, rows)], _slices(rows, few)):
        r, out = residual.clone(), torch.zeros((rows, width + padding), dtype=kind, device="cuda")
        for part in parts:
            assert call(_stream(), r[part].data_ptr(), change[part].data_ptr() if delta else None, width + padding,
                        out[part].data_ptr() if norm else None, width + padding, weight.data_ptr(), r[part].shape[0], width,
                        1e-5) == ks.OK
        results.append((r, out))
    torch.cuda.synchronize()
    assert all(torch.equal(*pair) for pair in zip(*results))


@pytest.mark.parametrize("index", [torch.int32, torch.int64])
@pytest.mark.parametrize("heads,kv_heads,dim,padding", [(32, 8, 128, 0), (5, 1, 16, 8), (6, 3, 64, 0), (33, 33, 32, 0), (2, 1, 512, 0),
                                                        (4, 2, 96, 0)])
def test_rotary_rows(index, heads, kv_heads, dim, padding):
    # (the last has a head of six lanes, which stays with the CTA per token)
    _, tokens, few = _counts()
    capacity, page = 300, 16
    gen = torch.Generator(device="cuda").manual_seed(dim)
    normal = lambda *shape: torch.randn(shape, generator=gen, device="cuda").to(torch.bfloat16)
    qkv, cosine, sine = normal(tokens, (heads + 2 * kv_heads) * dim + padding), normal(capacity, dim // 2), normal(capacity, dim // 2)
    pages = -(-tokens // page)
    place = torch.randperm(pages * page, generator=gen, device="cuda")[:tokens]
    position = torch.randint(-capacity, capacity, (tokens,), generator=gen, device="cuda").to(index)
    write_page, write_slot = (place // page).to(index), (place % page).to(index)
    write_page[1] -= pages          # wraps
    position[7] = capacity          # refused
    write_slot[9] = page            # its key and value are refused
    write_page[tokens - 1] = pages
    results = []
    for parts in ([slice(0, tokens)], _slices(tokens, few)):
        q = torch.zeros((tokens, heads, dim), dtype=torch.bfloat16, device="cuda")
        keys, values = (torch.zeros((pages, page, kv_heads, dim), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        for part in parts:
            assert ks.lib().singe_rotary_cache_write_bf16(
                _stream(), q[part].data_ptr(), qkv[part].data_ptr(), qkv.stride(0), cosine.data_ptr(), sine.data_ptr(),
                position[part].data_ptr(), keys.data_ptr(), values.data_ptr(), write_page[part].data_ptr(),
                write_slot[part].data_ptr(), position.element_size(), q[part].shape[0], heads, kv_heads, dim, pages, page, capacity,
                status.data_ptr()) == ks.OK
        results.append((q, keys, values, status))
    torch.cuda.synchronize()
    assert int(results[0][3].item()) == 1
    assert all(torch.equal(*pair) for pair in zip(*results))
