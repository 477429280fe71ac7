"""Where a query tile of the tcgen05 prompt attention (csrc/attention_prefill_tcgen05.cu) ends before its 128 rows or its last
block's 64 keys do, at both head sizes: rows that end inside a warp, and what lies where no row looks."""
from __future__ import annotations

import pytest
import torch

from test_attention_head_128_gpu import i32, plain

pytestmark = pytest.mark.gpu


def attention(dim, heads, groups, page, window, lengths, starts, unseen=0.0, seed=3):
    """(the kernel's output, the oracle's): random prompts in pages that lie anywhere but in page 0; page 0, pages of nobody and
    the places of a request's pages that it has not written hold ``unseen``."""
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)      # noqa: E731
    spans, tokens, scale = len(lengths), sum(lengths), dim ** -0.5
    needs = [-(-(s + n) // page) for s, n in zip(starts, lengths)]
    order = (1 + torch.randperm(sum(needs) + 2, generator=torch.Generator().manual_seed(1))).tolist()
    table = torch.full((spans, max(needs)), -1, dtype=torch.int32)
    caches = [torch.full((len(order) + 1, groups, page, dim), unseen, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    q, parts = rand(tokens, heads, dim), []
    for r, (start, n, need) in enumerate(zip(starts, lengths, needs)):
        pages = [order.pop() for _ in range(need)]
        at = torch.arange(start + n, device="cuda")
        where = torch.tensor(pages, device="cuda")[at // page]
        k, v = rand(start + n, groups, dim), rand(start + n, groups, dim)
        for cache, rows in zip(caches, (k, v)):
            cache[where, :, at % page] = rows
        table[r, :need] = torch.tensor(pages, dtype=torch.int32)
        if window and window > 0:                    # pages wholly before the window have been given back
            table[r, :max(0, start - window + 1) // page] = -1
        parts.append((k.double(), v.double()))
    positions = [p for s, n in zip(starts, lengths) for p in range(s, s + n)]
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    out, flag = torch.zeros(tokens, heads * dim, dtype=torch.bfloat16, device="cuda"), i32([0])
    kernels.attention_prefill_tcgen05(q.flatten(1), heads * dim, out, *caches, i32(positions), i32(begins), table.cuda(), tokens,
                                      spans, sum(-(-n // 128) for n in lengths), heads, groups, dim, page, window, scale, flag)
    assert int(flag.item()) == 0
    want = torch.cat([plain(q[a:b].double(), k, v, torch.tensor(positions[a:b], device="cuda"), scale, window, None, None, None)
                      for a, b, (k, v) in zip(begins, begins[1:], parts)]).flatten(1)
    return out.double(), want


@pytest.mark.parametrize("dim", [64, 128])
def test_rows_that_end_inside_a_warp(dim):
    """Spans whose last tile ends with 1, 31, 32, 33 .. live rows: every lane of a warp takes part in its loads from tensor
    memory, whichever of them store."""
    lengths = (1, 31, 32, 33, 63, 65, 95, 97, 127, 128, 129, 161)
    out, want = attention(dim, 8, 2, 16, None, lengths, tuple(7 * i for i in range(len(lengths))))
    # the weights and the output are rounded to 8 bits once each: two errors of at most 2^-9 of a row's numbers
    assert float((out - want).norm() / want.norm()) <= 2 ** -8


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("unseen", [float("nan"), float("inf")])
@pytest.mark.parametrize("page,window,lengths,starts", [
    (16, None, (5, 130, 200), (0, 3, 1000)), (8, 70, (129, 40), (500, 77)), (64, None, (33, 128), (0, 60)), (32, 150, (300,), (1001,)),
])
def test_places_that_no_row_of_a_tile_sees_may_hold_anything(dim, unseen, page, window, lengths, starts):
    """A weight of zero times a NaN is a NaN: what another request left in page 0, in a page that was used again or before the
    window does not reach a prompt's rows."""
    out, want = attention(dim, 4, 2, page, window, lengths, starts, unseen)
    # (as above)
    assert float((out - want).norm() / want.norm()) <= 2 ** -8
