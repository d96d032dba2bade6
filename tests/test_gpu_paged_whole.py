"""The Tensor surface's paged attention into uninitialised outputs against the same call into cleared ones."""
import pytest
import torch

from singe_b200 import kernel_sys as ks


pytestmark = pytest.mark.gpu

HEADS, KV_HEADS, PAGES = 8, 2, 40


def run(name, kind, fill, query, cache, offsets, page_offsets, pages, last, page_size, dim, index, with_status):
    tokens = query.shape[0]
    out = torch.full((tokens, HEADS, dim), fill[0], dtype=kind, device="cuda")
    lse = torch.full((tokens, HEADS), fill[1], device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lists = [torch.tensor(x, dtype=index, device="cuda") for x in (offsets, page_offsets, pages, last)]
    code = getattr(ks.lib(), name)(int(torch.cuda.current_stream().cuda_stream), out.data_ptr(), lse.data_ptr(), query.data_ptr(),
                                   cache[0].data_ptr(), cache[1].data_ptr(), *[x.data_ptr() for x in lists], lists[0].element_size(), tokens,
                                   HEADS, KV_HEADS, dim, page_size, PAGES, len(last), len(pages), dim ** -0.5, 1, 0,
                                   status.data_ptr() if with_status else None)
    torch.cuda.synchronize()
    assert code == ks.OK
    return out, lse, int(status.item())


# tokens, query offsets, page offsets (three pages a sequence), a page id that lies outside the cache or not
CASES = {"covered": (70, [0, 33, 34, 70], [0, 3, 6, 9], None), "gap in front": (70, [5, 33, 34, 70], [0, 3, 6, 9], None),
         "gap behind": (300, [0, 33, 34, 70], [0, 3, 6, 9], None), "refused page": (70, [0, 33, 34, 70], [0, 3, 6, 9], 1),
         "refused offsets": (70, [0, 33, 20, 70], [0, 3, 6, 9], None), "pages run backwards": (70, [0, 33, 34, 70], [0, 3, 2, 9], None),
         "one token each": (3, [0, 1, 2, 3], [0, 3, 6, 9], None), "one token each, refused": (3, [0, 1, 2, 3], [0, 3, 6, 9], 4),
         "no pages": (70, [0, 33, 34, 70], [0, 3, 3, 6], None)}


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("kind,page_size,dim", [(torch.bfloat16, 16, 128), (torch.bfloat16, 16, 64), (torch.bfloat16, 8, 64), (torch.float32, 16, 64)])
@pytest.mark.parametrize("index,with_status", [(torch.int64, True), (torch.int32, False)])
def test_whole_outputs(case, kind, page_size, dim, index, with_status):
    tokens, offsets, page_offsets, bad = CASES[case]
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    draw = lambda *shape: torch.randn(shape, generator=gen, device="cuda").to(kind)
    query, cache = draw(tokens, HEADS, dim), [draw(PAGES, page_size, KV_HEADS, dim) for _ in range(2)]
    pages = torch.randperm(PAGES, generator=torch.Generator().manual_seed(1))[: page_offsets[-1]].tolist()
    if bad is not None:
        pages[bad] = PAGES
    suffix = "bf16" if kind == torch.bfloat16 else "f32"
    rest = (query, cache, offsets, page_offsets, pages, [3, page_size, 1], page_size, dim, index, with_status)
    cleared = run(f"singe_paged_attention_{suffix}", kind, (0.0, float("-inf")), *rest)
    for fill in ((float("nan"), float("nan")), (7.0, 7.0)):
        whole = run(f"singe_paged_attention_whole_{suffix}", kind, fill, *rest)
        assert torch.equal(whole[0], cleared[0]) and torch.equal(whole[1], cleared[1]) and whole[2] == cleared[2]
