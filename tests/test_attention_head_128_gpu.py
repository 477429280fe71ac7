"""The tcgen05 attention for prompt portions at a head size of 128 (csrc/attention_prefill_tcgen05.cu) against float64: tiles
and blocks of keys that end early, rings that go round, pages of every size, masks, sinks, distance biases, capped scores, and
maxima that grow late (rescaled outputs)."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DIM = 128


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def plain(q, k, v, positions, scale, window, sinks, bias, softcap):
    """q [n, heads, 128] at `positions`, k, v [m, groups, 128]; float64."""
    heads, group = q.shape[1], q.shape[1] // k.shape[1]
    out = torch.empty_like(q)
    key = torch.arange(k.shape[0], device="cuda")[None]
    position = positions[:, None]
    seen = key <= position
    if window and window > 0:
        seen &= key > position - window
    elif window:
        seen &= key >= position - position % -window
    for h in range(heads):
        scores = q[:, h] @ k[:, h // group].T * scale
        if softcap:
            scores = softcap * torch.tanh(scores / softcap)
        if bias is not None:
            scores = scores + bias[h][(position - key).clamp(0, bias.shape[1] - 1)]
        scores = scores.masked_fill(~seen, -math.inf)
        if sinks is not None:
            scores = torch.cat([scores, sinks[h].expand(scores.shape[0], 1)], dim=1)
        out[:, h] = torch.softmax(scores, dim=-1)[:, :k.shape[0]] @ v[:, h // group]
    return out


@pytest.mark.parametrize("heads,groups,page,window,lengths,starts,extra", [
    (1, 1, 16, None, (128,), (0,), ""), (2, 1, 16, None, (1, 200), (0, 0), ""), (8, 2, 16, None, (130, 5, 77), (37, 0, 255), ""),
    (3, 3, 8, 150, (300,), (1000,), ""), (4, 4, 32, -100, (100, 260), (0, 40), ""), (6, 2, 64, 70, (129, 2), (500, 63), "sinks"),
    (2, 2, 16, None, (140,), (700,), "bias"), (4, 1, 16, 128, (90,), (333,), "softcap"), (2, 1, 16, None, (257,), (0,), "growing"),
])
def test_attention_of_head_size_128(heads, groups, page, window, lengths, starts, extra):
    from celeg_b200 import kernels
    assert kernels.attention_prefill_tcgen05_supported(heads, groups, DIM, page, torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)      # noqa: E731
    spans, tokens, scale = len(lengths), sum(lengths), DIM ** -0.5
    needs = [-(-(s + n) // page) for s, n in zip(starts, lengths)]
    order = torch.randperm(sum(needs) + 3, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((spans, max(needs)), -1, dtype=torch.int32)
    caches = [torch.full((len(order), groups, page, DIM), 1e4, device="cuda") for _ in range(2)]      # (unused pages: large)
    used, parts = 0, []
    q = rand(tokens, heads, DIM).to(torch.bfloat16)
    for r, (start, n, need) in enumerate(zip(starts, lengths, needs)):
        pages = order[used:used + need]
        used += need
        table[r, :need] = torch.tensor(pages, dtype=torch.int32)
        k, v = (rand(start + n, groups, DIM).to(torch.bfloat16).float() for _ in range(2))
        if extra == "growing":       # every block of keys has larger scores than the one before
            k *= (1 + 4 * torch.arange(start + n, device="cuda").div(64, rounding_mode="floor"))[:, None, None]
            k = k.to(torch.bfloat16).float()
        at = torch.arange(start + n, device="cuda")
        where = torch.tensor(pages, device="cuda")[at // page]
        for cache, rows in zip(caches, (k, v)):
            cache[torch.tensor(pages, device="cuda")] = 0.0
            cache[where, :, at % page] = rows
        parts.append((k.double(), v.double()))
    sinks = rand(heads) if extra == "sinks" else None
    bias = rand(heads, 60) if extra == "bias" else None
    softcap = 2.0 if extra == "softcap" else None
    positions = [p for s, n in zip(starts, lengths) for p in range(s, s + n)]
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    rows = torch.zeros(tokens + 5, heads * DIM + 72, dtype=torch.bfloat16, device="cuda")
    rows[:tokens, :heads * DIM] = q.flatten(1)
    out, flag = torch.zeros(tokens, heads * DIM, dtype=torch.bfloat16, device="cuda"), i32([0])
    kernels.attention_prefill_tcgen05(rows, rows.shape[1], out, caches[0].to(torch.bfloat16), caches[1].to(torch.bfloat16),
                                      i32(positions), i32(begins), table.cuda(), tokens, spans, sum(-(-n // 128) for n in lengths),
                                      heads, groups, DIM, page, window, scale, flag, sinks=sinks, distance_bias=bias, softcap=softcap)
    assert int(flag.item()) == 0
    want = torch.cat([plain(q[a:b].double(), k, v, torch.tensor(positions[a:b], device="cuda"), scale, window,
                            sinks.double() if sinks is not None else None, bias.double() if bias is not None else None, softcap)
                      for a, b, (k, v) in zip(begins, begins[1:], parts)]).flatten(1)
    # the weights and the output are rounded to 8 bits once each: two errors of at most 2^-9 of a row's numbers
    assert float((out.double() - want).norm() / want.norm()) <= 2 ** -8
