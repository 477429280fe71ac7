"""The forms of the chunked scans that their rules select, each against float64: the walk over the chunks with 32 and with 64 columns
a block, sums of the chunks side by side, the delta rules' walk with 32 columns a block (from 149 blocks of 16 on), read-outs of one
to eight heads a block; and the delta rules' mixers on single tokens and portions in one step."""
from __future__ import annotations

import pytest
import torch

import test_chunk_scan_gpu as chunk_scan
from test_chunk_scan_gpu import i32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,heads,kv_heads,dim,vdim,slowest", [
    ([130], 40, 20, 64, 64, 1e-3),                   # 160 blocks of 16 columns
    ([70, 65], 19, 19, 40, 70, 1e-2),                # 190, the last block of a head almost empty; a key size between tiles
    ([100], 20, 20, 128, 128, 1e-3),                 # 160 of wide keys
    ([66, 129], 19, 19, 72, 60, 0.1),                # 152 of wide keys, a size between tiles
])
def test_delta_rule_with_32_columns_a_block(lengths, heads, kv_heads, dim, vdim, slowest):
    assert -(-vdim // 16) * heads * len(lengths) > 148
    chunk_scan.test_delta_rule_in_chunks_is_as_near_to_64_bits_as_token_by_token(lengths, heads, kv_heads, dim, vdim, slowest)


@pytest.mark.parametrize("lengths,heads,dim", [([130], 40, 64), ([70, 65], 30, 40)])
def test_generalised_delta_rule_with_32_columns_a_block(lengths, heads, dim):
    assert -(-dim // 16) * heads * len(lengths) > 148
    chunk_scan.test_generalised_delta_rule_in_chunks_of_64(lengths, heads, dim, 0.0)


def linear(begins, q, k, v, decay, before):
    """float64: (read-outs, states) of S <- diag(decay) S + k v^T, o = S^T q; q, k, v, decay [tokens, heads, ..]."""
    out, after = torch.zeros_like(v), before.double().clone()
    for span in range(len(begins) - 1):
        for t in range(begins[span], begins[span + 1]):
            after[span] = decay[t].unsqueeze(-1) * after[span] + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
            out[t] = (after[span] * q[t].unsqueeze(-1)).sum(-2)
    return out.flatten(1), after


@pytest.mark.parametrize("kind,lengths,heads,groups,dim,vdim,columns,share", [
    ("scalar", [130], 100, 100, 64, 64, 64, 1),              # (no heads share keys)
    ("scalar", [64 * 9 + 1, 63], 64, 8, 64, 33, 0, 2),
    ("scalar", [64 * 19 + 5], 64, 8, 72, 20, 32, 2),
    ("scalar", [900], 64, 8, 72, 20, 32, 4),
    ("scalar", [2048], 64, 8, 128, 64, 64, 8),
    ("scalar", [100, 64], 64, 8, 64, 33, 64, 1),             # one column in the second half of a block's 64
    ("channel", [63, 64, 65], 40, 40, 40, 50, 64, 1), ("channel", [70], 60, 60, 136, 33, 32, 1), ("channel", [130, 64], 2, 2, 40, 33, 0, 1),
    ("constant", [100, 64], 120, 120, 40, 70, 32, 1),
    ("constant", [65, 130], 64, 64, 64, 33, 64, 1), ("constant", [70], 60, 60, 136, 33, 32, 1),
    ("constant", [70, 193, 128], 2, 2, 136, 70, 0, 1),       # queries in two passes
    ("constant", [577, 1, 1, 64], 16, 16, 40, 66, 0, 1),     # one long span beside short ones
])
def test_walk_and_shared_read_outs(kind, lengths, heads, groups, dim, vdim, columns, share):
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(23)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)      # noqa: E731
    full = lambda *shape: torch.full(shape, 5.0, device="cuda")                # noqa: E731
    tokens, spans, wide, elements = sum(lengths), len(lengths), heads * vdim, heads * dim * vdim
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    chunks = tokens // 64 + spans
    cut = 2 * (tokens // 128 + spans) if kind == "constant" else chunks
    assert kernels.chunk_walk_columns(False, heads, dim, vdim, spans, cut, max(lengths)) == columns
    assert kind != "scalar" or kernels.chunk_read_heads(heads, groups, dim, vdim, chunks) == share
    q, k, v = rand(tokens, groups * dim), rand(tokens, groups * dim), rand(tokens, wide)
    before, out = rand(spans, elements), full(tokens, wide)
    state = before.clone()
    plan = torch.zeros(2 * chunks + spans + 16, dtype=torch.int32, device="cuda")
    kernels.chunk_plan(i32(begins), spans, chunks + 3, plan)
    slots = i32(list(range(spans)))
    where = (state, state.stride(0), slots, plan, chunks + 3, spans, chunks)
    q64, k64, v64 = q.double().view(tokens, groups, dim), k.double().view(tokens, groups, dim), v.double().view(tokens, heads, vdim)
    if kind == "scalar":
        raw, a_log, direct, bias = rand(tokens, heads), rand(heads) - 2, rand(heads), rand(heads) - 2
        kernels.scalar_decay_scan(q, k, v, raw, bias, a_log, direct, full(tokens, 2 * heads), full(tokens, heads), None,
                                  full(chunks * elements), out, *where, heads, groups, dim, vdim, max(lengths))
        dt = torch.nn.functional.softplus((raw + bias).double(), threshold=100.0)
        share = heads // groups
        want, want_state = linear(begins, q64.repeat_interleave(share, 1), k64.repeat_interleave(share, 1) * dt.unsqueeze(-1), v64,
                                  torch.exp(-torch.exp(a_log.double()) * dt).unsqueeze(-1), before.view(spans, heads, dim, vdim))
        want = want + (direct.double()[:, None] * v64).flatten(1)
    elif kind == "channel":
        z, bias = rand(tokens, heads * dim), rand(heads * dim)
        kernels.channel_decay_scan(q, k, v, z, bias, 16.0, 0.3, full(tokens, heads * dim), full(tokens, heads * dim),
                                   full(chunks * heads * dim), full(chunks * heads * 4096), full(chunks * elements), out, *where, heads,
                                   dim, vdim, max(lengths))
        decay = torch.exp(torch.nn.functional.logsigmoid((z + bias).double()) / 16.0).view(tokens, heads, dim)
        want, want_state = linear(begins, q64 * 0.3, k64, v64, decay, before.view(spans, heads, dim, vdim))
    else:
        decay = 1.0 - 2.0 ** (-2.0 - 6.0 * torch.rand(heads, device="cuda", generator=g))
        segments = tokens // 128 + spans
        kernels.retention_segmented(q, k, v, decay, out, state, state.stride(0), i32(begins), slots, spans, tokens, heads, dim, vdim,
                                    0.3, 128, segments, full(2 * segments * elements),
                                    torch.zeros(segments + spans + 2, dtype=torch.int32, device="cuda"), longest=max(lengths))
        each = decay.double().view(1, heads, 1).expand(tokens, heads, 1)
        want, want_state = linear(begins, q64, k64 * 0.3, v64, each, before.view(spans, heads, dim, vdim))
    # a weight is a product of up to 64 decays with a rounding each: 64 units of 2^-24 at most
    for name, a, b in (("read", out, want), ("state", state, want_state.flatten(1))):
        off = float((a.double() - b).norm() / b.norm())
        assert off <= 64 * 2 ** -24, (name, off)


@pytest.mark.parametrize("lengths,heads,dim,vdim,forget,columns", [
    ([70, 300], 40, 64, 96, -3.0, 64),               # a decay of a twentieth a token
    ([100, 64], 64, 64, 128, 2.0, 32),               # two spans of two chunks, whole blocks
    ([63, 64, 65], 40, 40, 33, 3.0, 64),             # odd columns
    ([70, 65, 64, 1], 40, 136, 33, 1.0, 32),         # three blocks of key channels, the last one almost empty
    ([130], 100, 72, 20, 4.0, 32),                   # a head in less than half of a block
    ([577, 1, 64], 6, 32, 48, 3.0, 0),               # one long span beside short ones
])
def test_mlstm_by_either_route(lengths, heads, dim, vdim, forget, columns):
    from celeg_b200 import kernels
    chunks = sum(lengths) // 64 + len(lengths)
    assert kernels.chunk_walk_columns(True, heads, dim, vdim, len(lengths), chunks, max(lengths)) == columns
    chunk_scan.test_mlstm_in_chunks_is_as_near_to_64_bits_as_token_by_token(lengths, heads, dim, vdim, forget)


@pytest.mark.parametrize("stable", [False, True])
def test_one_long_span_beside_short_ones_is_not_walked(stable):
    """The walk takes a span's chunks one after another: with a span of 4,096 tokens beside seven of 64, or of 3,500 beside fifteen
    of 40, it takes two to three times what the sums do."""
    from celeg_b200 import kernels
    for lengths in ([4096] + [64] * 7, [3500] + [40] * 15):
        chunks = sum(lengths) // 64 + len(lengths)
        for heads, dim, vdim in ((16, 64, 128), (16, 128, 64), (8, 96, 96)):
            assert kernels.chunk_walk_columns(stable, heads, dim, vdim, len(lengths), chunks, max(lengths)) == 0
    assert kernels.chunk_walk_columns(stable, 16, 64, 128, 16, 53, 150) != 0        # sixteen of 150


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["gated_delta", "general_delta"])
def test_delta_mixers_on_single_tokens_and_portions_together(kind, dtype):
    """Two single tokens, a long portion (chunks) and a short one in one step give what they give token by token."""
    from celeg_b200.parts import Runtime, StateBinding, StepContext, part_factory
    g = torch.Generator().manual_seed(6)
    hidden, heads, kv, dim, vdim, rows = 48, 4, 2, 16, 24, 576
    matrix = lambda n, m: (torch.randn(n, m, generator=g) * m ** -0.5).to(torch.bfloat16)        # noqa: E731
    vector = lambda n, mean=0.0: (mean + 0.3 * torch.randn(n, generator=g)).to(torch.bfloat16)   # noqa: E731
    params = {"hidden_size": hidden, "heads": heads, "dim": dim, "vdim": vdim, "kv_heads": kv, "taps": 4, "eps": 1e-5}
    if kind == "gated_delta":
        weights = {"q": matrix(kv * dim, hidden), "k": matrix(kv * dim, hidden), "v": matrix(heads * vdim, hidden),
                   "gate": matrix(heads * vdim, hidden), "beta": matrix(heads, hidden), "decay": matrix(heads, hidden),
                   "q_conv": matrix(kv * dim, 4), "k_conv": matrix(kv * dim, 4), "v_conv": matrix(heads * vdim, 4),
                   "a_log": vector(heads, -1.0), "dt_bias": vector(heads), "norm": vector(vdim, 1.0), "out": matrix(hidden, heads * vdim)}
    else:
        inner = heads * dim
        weights = {n: matrix(inner, hidden) for n in ("r", "k", "v", "gate", "removal")}
        weights.update({"decay_down": matrix(8, hidden), "decay_up": matrix(inner, 8), "removal_bias": vector(inner),
                        "decay_bias": vector(inner), "norm": vector(inner, 1.0), "out": matrix(hidden, inner)})
    lengths = [1, 1, 520, 3]
    tokens, begins = sum(lengths), [0, 1, 2, 522, 525]
    x = torch.zeros(rows, hidden, dtype=dtype, device="cuda")
    x[:tokens] = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    results = []
    for chunked in (True, False):
        rt = Runtime(torch.device("cuda:0"), dtype, rows, max_requests=8, max_context=1024)
        mixer = part_factory("mixer", kind)(params, weights, {}, rt)
        if not chunked:
            mixer.CHUNKED_FROM = 10 ** 9
        assert mixer.in_chunks(lengths[2:]) == chunked
        elements = mixer.cache_need().elements
        state = torch.full((5, -(-elements // 4) * 4), 0.25, device="cuda")
        mixer.bind_cache(StateBinding(state=state, slot_stride=state.stride(0)))
        step = StepContext(tokens=tokens, spans=4, token_ids=i32([0] * tokens), positions=i32(list(range(tokens))),
                           token_span=i32([i for i, n in enumerate(lengths) for _ in range(n)]), span_begin=i32(begins),
                           span_slot=i32([3, 0, 4, 1]), block_tables=[], error_flag=torch.zeros(1, dtype=torch.int32, device="cuda"),
                           max_span=520, max_context=520, context_bucket=1024, host_span_lengths=lengths, leading_single_tokens=2)
        out = torch.zeros_like(x)
        mixer.forward(x, out, step)
        assert int(step.error_flag.item()) == 0
        results.append((out[:tokens].double(), state.double()))
    # float32: order of sums; bfloat16: the gated read-outs and the output are rounded once more, to 8 bits
    bound = 2e-5 if dtype == torch.float32 else 2 ** -8
    for a, b in zip(*results):
        assert float((a - b).norm() / b.norm()) <= bound


@pytest.mark.parametrize("spread,repeat", [(0.0, 1), (0.05, 1), (0.05, 3)])
@pytest.mark.parametrize("decay", [-8.0, 0.0])
def test_generalised_delta_rule_with_keys_that_resemble_one_another(spread, repeat, decay):
    """Equal or nearly equal keys, in turn ``repeat`` of them, a decay of almost one or of about 0.7: what is written and what is
    removed again nearly cancel, more of it in a chunk of 64 tokens than in one of eight."""
    import math
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(29)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)      # noqa: E731
    full = lambda *shape: torch.full(shape, 5.0, device="cuda")                # noqa: E731
    tokens, heads, dim, eps = 512, 4, 64, 1e-6
    inner, chunks = heads * dim, tokens // 64 + 1
    proj, z, w0, a_bias = rand(tokens, 4 * inner), rand(tokens, inner) + decay, rand(inner) * 0.3, rand(inner) * 0.3
    offsets = (0, inner, 2 * inner, 3 * inner)
    proj[:, inner:2 * inner] = rand(repeat, inner).repeat(-(-tokens // repeat), 1)[:tokens] + spread * proj[:, inner:2 * inner]
    before, begins, slots, flag = rand(1, inner * dim), i32([0, tokens]), i32([0]), i32([0])
    r, k, v, a = (proj[:, o:o + inner].double().view(tokens, heads, dim) for o in offsets)
    keep = torch.exp(-math.exp(-0.5) * torch.sigmoid((z + w0).double())).view(tokens, heads, dim)
    unit = k / torch.sqrt(k.square().sum(-1, keepdim=True) + eps)
    removal = torch.sigmoid(a + a_bias.double().view(heads, dim)) * unit
    s, want = before[0].double().view(heads, dim, dim), torch.zeros(tokens, heads, dim, device="cuda", dtype=torch.float64)
    for t in range(tokens):
        taken = (s * unit[t].unsqueeze(-1)).sum(-2)
        s = keep[t].unsqueeze(-1) * s - removal[t].unsqueeze(-1) * taken.unsqueeze(-2) + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
        want[t] = (s * r[t].unsqueeze(-1)).sum(-2)
    by_eight, eight_state = full(tokens, inner), before.clone()
    kernels.general_delta_scan(proj, offsets, z, w0, a_bias, eps, i32([0] * tokens), begins, slots,
                               torch.zeros(tokens * kernels.general_delta_scratch(heads, dim), device="cuda"), by_eight, eight_state,
                               before.stride(0), tokens, 1, heads, dim, flag)
    got, got_state = full(tokens, inner), before.clone()
    plan = torch.zeros(2 * chunks + 16, dtype=torch.int32, device="cuda")
    kernels.chunk_plan(begins, 1, chunks + 3, plan)
    kernels.general_delta_chunk_scan(proj, offsets, z, w0, a_bias, eps, full(tokens, inner), full(chunks * heads * 4096),
                                     full(chunks * heads * 4096), full(chunks * heads * kernels.delta_operand_bytes(dim) // 4),
                                     full(tokens, inner), full(chunks * inner * dim), full(chunks * inner), got, got_state,
                                     before.stride(0), slots, plan, chunks + 3, 1, chunks, heads, dim, flag)
    assert int(flag.item()) == 0
    off = lambda x, y: float((x.double() - y).norm() / y.norm())               # noqa: E731
    # the same size of error as in chunks of eight, and a state's element passes through three roundings more at its end
    for a, b, c in ((got, by_eight, want.flatten(1)), (got_state, eight_state, s.flatten()[None])):
        assert off(a, c) <= 1.5 * off(b, c) + 3 * 2 ** -24, (off(a, c), off(b, c))
