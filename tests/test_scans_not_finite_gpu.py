"""Decays of zero, and what a NaN in one token's rows does, in the chunked scans (csrc/chunk_scan.cuh, csrc/delta_chunks.cu): the tokens before it,
other heads, other requests and, for a value, other columns are bit for bit what they are without it; the head's (or the
column's) read-outs from that token on and the state afterwards are NaN, as token by token."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS, HEADS, DIM = (70, 40, 129), 2, 40
BEGINS = (0, 70, 110, 239)
TOKENS, SPANS = 239, 3
CHUNKS = TOKENS // 64 + SPANS


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def full(*shape):
    return torch.full(shape, 5.0, device="cuda")


def scan(kind, x, vdim):
    """(read-outs [tokens, heads, vdim], states [spans, heads, dim, vdim]) of one chunked scan; x: its inputs by name."""
    from celeg_b200 import kernels
    wide, elements = HEADS * vdim, HEADS * DIM * vdim
    out, state = full(TOKENS, wide), torch.full((SPANS, elements + HEADS * (DIM + 1)), 0.25, device="cuda")
    begins, slots, flag = i32(BEGINS), i32([2, 0, 1]), i32([0])
    plan = torch.zeros(2 * (CHUNKS + 3) + 16, dtype=torch.int32, device="cuda")
    kernels.chunk_plan(begins, SPANS, CHUNKS + 3, plan)
    states = full(CHUNKS * elements)
    where = (state, state.stride(0), slots, plan, CHUNKS + 3, SPANS, CHUNKS)
    gate, rate, ones = x["gate"], x["rate"], torch.ones(HEADS, device="cuda")
    operands = full(CHUNKS * HEADS * kernels.delta_operand_bytes(DIM) // 4)
    if kind == "mlstm":
        kernels.mlstm_chunk_scan(x["q"], x["k"], x["v"], gate[:, :HEADS], gate[:, HEADS:], -ones, 3 * ones, 15.0,
                                 full(TOKENS, 6 * HEADS), torch.zeros(CHUNKS * HEADS, dtype=torch.float64, device="cuda"),
                                 full(CHUNKS * HEADS * DIM), states, out, *where, HEADS, DIM, vdim, 0.2)
    elif kind == "retention":
        kernels.retention_segmented(x["q"], x["k"], x["v"], torch.tensor([0.9, 0.97], device="cuda"), out, state, state.stride(0),
                                    begins, slots, SPANS, TOKENS, HEADS, DIM, vdim, 0.2, 128, TOKENS // 128 + SPANS,
                                    full(2 * (TOKENS // 128 + SPANS) * elements), torch.zeros(32, dtype=torch.int32, device="cuda"),
                                    torch.arange(16, dtype=torch.int32, device="cuda"))
    elif kind == "gated_delta":
        k = torch.nn.functional.normalize(x["k"].view(TOKENS, HEADS, DIM), dim=-1).view(TOKENS, -1)
        kernels.delta_chunk_scan(x["q"], k, x["v"], torch.sigmoid(gate), rate, ones, ones, full(TOKENS, 2 * HEADS),
                                 full(TOKENS, HEADS), operands, full(TOKENS, wide), states, out, *where, HEADS, HEADS, DIM, vdim,
                                 0.2, flag)
    elif kind == "general_delta":
        inner = HEADS * DIM
        proj = torch.cat([x["q"], x["k"], x["v"], x["a"]], dim=1)
        kernels.general_delta_chunk_scan(proj, (0, inner, 2 * inner, 3 * inner), x["z"], torch.zeros(inner, device="cuda"),
                                         torch.zeros(inner, device="cuda"), 1e-6, full(TOKENS, inner), full(CHUNKS * HEADS * 4096),
                                         full(CHUNKS * HEADS * 4096), operands, full(TOKENS, inner), states, full(CHUNKS * inner),
                                         out, *where, HEADS, DIM, flag)
    elif kind == "gated_linear_attention":
        inner = HEADS * DIM
        kernels.channel_decay_scan(x["q"], x["k"], x["v"], x["z"], torch.zeros(inner, device="cuda"), 16.0, 0.2, full(TOKENS, inner),
                                   full(TOKENS, inner), full(CHUNKS * inner), full(CHUNKS * HEADS * 4096), states, out, *where,
                                   HEADS, DIM, vdim)
    elif kind == "mamba2":
        kernels.scalar_decay_scan(x["q"], x["k"], x["v"], rate, -ones, ones, ones, full(TOKENS, 2 * HEADS), full(TOKENS, HEADS),
                                  full(CHUNKS * HEADS * 4096), states, out, *where, HEADS, HEADS, DIM, vdim)
    assert int(flag.item()) == 0
    return out.view(TOKENS, HEADS, vdim), state[:, :elements].view(SPANS, HEADS, DIM, vdim)[[2, 0, 1]]


# (linear attention's decays are taken apart in blocks of eight tokens: a NaN there reaches its block)
USES = {"mlstm": ("v", "k", "gate"), "retention": ("v", "k"), "gated_delta": ("v", "k", "gate", "rate"),
        "general_delta": ("v", "k", "a", "z"), "gated_linear_attention": ("v", "k"), "mamba2": ("v", "k", "rate")}


@pytest.mark.parametrize("at", [0, 5, 37, 66, 100, 200])
@pytest.mark.parametrize("kind,what", [(kind, what) for kind, names in USES.items() for what in names])
def test_a_nan_reaches_its_own_token_and_those_behind_it(kind, what, at):
    vdim = DIM if kind == "general_delta" else 70
    g = torch.Generator(device="cuda").manual_seed(17)
    rand = lambda columns: torch.randn(TOKENS, columns, device="cuda", generator=g)      # noqa: E731
    x = {"q": rand(HEADS * DIM), "k": rand(HEADS * DIM), "v": rand(HEADS * vdim), "gate": rand(2 * HEADS), "rate": rand(HEADS),
         "a": rand(HEADS * DIM), "z": rand(HEADS * DIM)}
    clean, clean_state = scan(kind, x, vdim)
    columns = {"v": vdim, "k": DIM, "a": DIM, "z": DIM, "gate": 1, "rate": 1}[what]
    column = min(33, columns - 1)
    x[what] = x[what].clone()
    x[what][at, columns + column] = float("nan")                               # of the second head
    got, got_state = scan(kind, x, vdim)
    span = next(s for s in range(SPANS) if at < BEGINS[s + 1])
    expected, expected_state = clean.clone(), clean_state.clone()
    reach = slice(column, column + 1) if what == "v" else slice(None)
    nan = float("nan")
    expected[at:BEGINS[span + 1], 1, reach] = nan
    expected_state[span, 1, :, reach] = nan
    if kind != "general_delta" and kind != "gated_delta" and what == "k":      # a key's channel is a row of the state
        expected_state[span] = clean_state[span]
        expected_state[span, 1, column] = nan
    same = (got == expected) | (got.isnan() & expected.isnan())
    assert bool(same.all()), (~same).nonzero()[:8].tolist()
    same = (got_state == expected_state) | (got_state.isnan() & expected_state.isnan())
    assert bool(same.all()), (~same).nonzero()[:8].tolist()


@pytest.mark.parametrize("rate,step", [(85.0, 0.0), (100.0, 0.0), (0.0, 3e30), (0.0, float("inf")), (30.0, 1e20)])
def test_a_decay_of_zero_leaves_the_decays_behind_it_alone(rate, step):
    """exp(-exp(a_log) softplus(.)) with logarithms from -1e13 to minus infinity, at some tokens or at all of them: the old state
    is gone there, and what follows decays as it does without them."""
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(19)
    rand = lambda columns: torch.randn(TOKENS, columns, device="cuda", generator=g)      # noqa: E731
    q, v, pre_a, dim, vdim = rand(HEADS * DIM), rand(HEADS * 24), rand(HEADS), DIM, 24
    k = torch.nn.functional.normalize(rand(HEADS * DIM).view(TOKENS, HEADS, DIM), dim=-1).view(TOKENS, -1)
    if step:
        pre_a[[3, 70, 71, 150], 1] = step
    a_log, dt_bias = torch.tensor([-2.0, rate], device="cuda"), torch.zeros(HEADS, device="cuda")
    decay = torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(pre_a, threshold=30.0))
    gates = torch.cat([torch.sigmoid(rand(HEADS)), decay], dim=1).contiguous()
    assert bool(gates.isfinite().all()) and float(decay.min()) == 0.0
    begins, slots, flag = i32(BEGINS), i32([2, 0, 1]), i32([0])
    before = torch.full((SPANS, HEADS * dim * vdim), 0.25, device="cuda")
    want, want_state = full(TOKENS, HEADS * vdim), before.clone()
    kernels.recurrent_scan(kernels.SCAN_DELTA, q, k, v, gates, want, want_state, before.stride(0), begins, slots, SPANS, HEADS, HEADS,
                           dim, vdim, 0.2)
    plan = torch.zeros(2 * (CHUNKS + 3) + 16, dtype=torch.int32, device="cuda")
    kernels.chunk_plan(begins, SPANS, CHUNKS + 3, plan)
    got, got_state = full(TOKENS, HEADS * vdim), before.clone()
    kernels.delta_chunk_scan(q, k, v, gates, pre_a, dt_bias, a_log, full(TOKENS, 2 * HEADS), full(TOKENS, HEADS),
                             full(CHUNKS * HEADS * kernels.delta_operand_bytes(dim) // 4), full(TOKENS, HEADS * vdim),
                             full(CHUNKS * HEADS * dim * vdim), got, got_state, before.stride(0), slots, plan, CHUNKS + 3, SPANS, CHUNKS,
                             HEADS, HEADS, dim, vdim, 0.2, flag)
    assert int(flag.item()) == 0
    # float32 sums of the same products in two orders, behind decays that differ in their last bits: a few units of 2^-24
    for a, b in ((got, want), (got_state, want_state)):
        assert float((a.double() - b.double()).norm() / b.double().norm()) <= 2e-6
