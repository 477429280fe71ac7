"""The mLSTM and the gated delta rule in chunks (csrc/chunk_scan.cuh, csrc/delta_chunks.cu) against a float64 restatement and
the token-by-token kernels, at the edges of chunks (64 tokens), of the blocks of key channels (32, 64, 128) and of columns (32,
64), and the mLSTM's mixer on a step of single tokens and portions."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def plain_mlstm(q, k, v, gate_i, gate_f, state, begins, slots, heads, dim, vdim):
    """float64: (read-outs [tokens, heads, vdim], the slots afterwards); rows of ``state``: S, normalisers, maxima."""
    q, k, v = q.double().view(-1, heads, dim) * dim ** -0.5, k.double().view(-1, heads, dim), v.double().view(-1, heads, vdim)
    out, after = torch.zeros_like(v), state.double().clone()
    s_end, n_end = heads * dim * vdim, heads * dim * (vdim + 1)
    for span, slot in enumerate(slots):
        row = after[slot]
        s, n, m = row[:s_end].view(heads, dim, vdim).clone(), row[s_end:n_end].view(heads, dim).clone(), row[n_end:n_end + heads].clone()
        for t in range(begins[span], begins[span + 1]):
            peak = torch.maximum(gate_f[t] + m, gate_i[t])
            keep, write, m = torch.exp(gate_f[t] + m - peak), torch.exp(gate_i[t] - peak), peak
            s = keep[:, None, None] * s + (write[:, None] * k[t]).unsqueeze(-1) * v[t].unsqueeze(-2)
            n = keep[:, None] * n + write[:, None] * k[t]
            out[t] = (s * q[t].unsqueeze(-1)).sum(-2) / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
        row[:s_end], row[s_end:n_end], row[n_end:n_end + heads] = s.flatten(), n.flatten(), m
    return out.flatten(1), after


@pytest.mark.parametrize("lengths,heads,dim,vdim,forget", [
    ([64, 65, 1, 128, 63], 3, 24, 36, 0.0),          # whole chunks, one token more and less; sizes between tiles
    ([200], 2, 64, 128, 5.0),                        # a normal head, almost nothing forgotten
    ([130, 66], 2, 40, 7, 2.0),                      # odd columns: no access of two or four
    ([97], 1, 130, 64, 3.0),                         # two blocks of key channels, one almost empty
    ([70, 300], 40, 64, 96, -3.0),                   # blocks of many heads; a decay of a twentieth a token
])
def test_mlstm_in_chunks_is_as_near_to_64_bits_as_token_by_token(lengths, heads, dim, vdim, forget):
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(11)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)      # noqa: E731
    tokens, spans, cap = sum(lengths), len(lengths), 15.0
    rows = rand(tokens, heads * (2 * dim + vdim) + 2 * heads + 3)              # as a projection's rows: one stride
    q, k = rows[:, :heads * dim], rows[:, heads * dim:2 * heads * dim]
    v = rows[:, 2 * heads * dim:heads * (2 * dim + vdim)]
    pre_i, pre_f = rows[:, heads * (2 * dim + vdim):][:, :heads], rows[:, heads * (2 * dim + vdim) + heads:][:, :heads]
    bias_i, bias_f = rand(heads) - 2, rand(heads) + forget
    elements = heads * dim * (vdim + 1) + heads
    before = rand(spans + 1, elements + 5)
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    slots = list(range(spans, 0, -1))
    gate_i = cap * torch.tanh((pre_i.double() + bias_i) / cap)
    gate_f = torch.nn.functional.logsigmoid(cap * torch.tanh((pre_f.double() + bias_f) / cap))
    want, want_state = plain_mlstm(q, k, v, gate_i, gate_f, before, begins, slots, heads, dim, vdim)

    gates, out, state = torch.zeros(tokens, 2 * heads, device="cuda"), torch.zeros(tokens, heads * vdim, device="cuda"), before.clone()
    kernels.mlstm_gates(pre_i, pre_f, bias_i, bias_f, cap, gates, tokens, heads)
    kernels.recurrent_scan(kernels.SCAN_MLSTM, q, k, v, gates, out, state, state.stride(0), i32(begins), i32(slots), spans, heads,
                           heads, dim, vdim, dim ** -0.5)
    chunks = tokens // 64 + spans
    full = lambda *shape: torch.full(shape, 5.0, device="cuda")                # noqa: E731
    plan, got, got_state = torch.zeros(chunks + spans + 8, dtype=torch.int32, device="cuda"), full(tokens, heads * vdim), before.clone()
    kernels.chunk_plan(i32(begins), spans, chunks + 3, plan)
    kernels.mlstm_chunk_scan(q, k, v, pre_i, pre_f, bias_i, bias_f, cap, full(tokens, 6 * heads),
                             torch.zeros(chunks * heads, dtype=torch.float64, device="cuda"), full(chunks * heads * dim),
                             full(chunks * heads * dim * vdim), got, got_state, got_state.stride(0), i32(slots), plan, chunks + 3,
                             spans, chunks, heads, dim, vdim, dim ** -0.5, max(lengths))

    def off(x, y):
        return float((x.double() - y).norm() / y.norm())
    # both are float32 sums of the same products in different orders: errors of the same size, of a few units of 2^-24
    for name, a, b, c in (("read", got, out, want), ("state", got_state, state, want_state)):
        assert off(a, c) <= 2 * off(b, c) + 3e-7, (name, off(a, c), off(b, c))
    assert torch.equal(got_state[:, elements:], before[:, elements:]) and torch.equal(got_state[0], before[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_mlstm_mixer_on_single_tokens_and_portions_together(dtype):
    """Two single tokens, a long portion (chunks) and a short one in one step give what they give alone, token by token."""
    from celeg_b200.parts import Runtime, StateBinding, StepContext, part_factory
    g = torch.Generator().manual_seed(5)
    hidden, heads, dim, vdim = 48, 2, 16, 24
    shapes = {"q": heads * dim, "k": heads * dim, "v": heads * vdim, "gate": heads * vdim, "input_gate": heads, "forget_gate": heads}
    weights = {n: (torch.randn(rows, hidden, generator=g) * hidden ** -0.5).to(torch.bfloat16) for n, rows in shapes.items()}
    weights.update({"out": torch.randn(hidden, heads * vdim, generator=g).to(torch.bfloat16),
                    "norm": torch.ones(heads * vdim), "input_gate_bias": torch.zeros(heads), "forget_gate_bias": torch.full((heads,), 3.0)})
    params = {"hidden_size": hidden, "heads": heads, "dim": dim, "vdim": vdim, "gate_cap": 15.0, "eps": 1e-5}
    lengths = [1, 1, 140, 3]
    tokens = sum(lengths)
    x = torch.zeros(192, hidden, dtype=dtype, device="cuda")
    x[:tokens] = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    results = []
    for chunked_from in (96, 10 ** 9):
        rt = Runtime(torch.device("cuda:0"), dtype, 192, max_requests=8, max_context=256)
        mixer = part_factory("mixer", "mlstm")(params, weights, {}, rt)
        mixer.CHUNKED_FROM = chunked_from
        elements = mixer.cache_need().elements
        state = torch.full((5, elements), 0.25, device="cuda")
        mixer.bind_cache(StateBinding(state=state, slot_stride=state.stride(0)))
        begins = [0, 1, 2, 142, 145]
        step = StepContext(tokens=tokens, spans=4, token_ids=i32([0] * tokens), positions=i32(list(range(tokens))),
                           token_span=i32([i for i, n in enumerate(lengths) for _ in range(n)]), span_begin=i32(begins),
                           span_slot=i32([3, 0, 4, 1]), block_tables=[], error_flag=torch.zeros(1, dtype=torch.int32, device="cuda"),
                           max_span=140, max_context=140, context_bucket=256, host_span_lengths=lengths, leading_single_tokens=2)
        out = torch.zeros_like(x)
        mixer.forward(x, out, step)
        results.append((out[:tokens].double(), state.double()))
    # float32: order of sums; bfloat16: the gated read-outs and the output are rounded once more, to 8 bits
    bound = 2e-5 if dtype == torch.float32 else 2 ** -8
    for a, b in zip(*results):
        assert float((a - b).norm() / b.norm()) <= bound


@pytest.mark.parametrize("lengths,heads,kv_heads,dim,vdim,slowest", [
    ([64, 65, 1, 128, 63], 4, 2, 24, 36, 1e-3),      # whole chunks, one token more and less; shared keys; sizes between tiles
    ([200], 2, 2, 64, 64, 1e-4),                     # a normal head, almost nothing forgotten
    ([130, 66], 2, 1, 40, 7, 0.1),                   # odd columns: no access of two or four
    ([97], 3, 3, 128, 200, 1e-2),                    # wide keys, more right sides than a pass of the solver takes
    ([70, 150], 2, 1, 66, 32, 3.0),                  # just beyond 64 keys; decays of a twentieth a token
])
def test_delta_rule_in_chunks_is_as_near_to_64_bits_as_token_by_token(lengths, heads, kv_heads, dim, vdim, slowest):
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(12)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)      # noqa: E731
    tokens, spans = sum(lengths), len(lengths)
    rows = rand(tokens, kv_heads * 2 * dim + heads * vdim + 5)                 # as the prepared rows: one stride
    q, k = rows[:, :kv_heads * dim], rows[:, kv_heads * dim:2 * kv_heads * dim]
    for part in (q, k):
        part.copy_(torch.nn.functional.normalize(part.reshape(tokens, kv_heads, dim), dim=-1).reshape(tokens, -1))
    v = rows[:, 2 * kv_heads * dim:2 * kv_heads * dim + heads * vdim]
    pre_a, dt_bias, a_log = rand(tokens, heads), rand(heads), torch.full((heads,), slowest, device="cuda").log()
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus((pre_a + dt_bias).double(), threshold=100.0))
    gates = torch.cat([torch.sigmoid(rand(tokens, heads)), decay.float()], dim=1).contiguous()
    elements = heads * dim * vdim
    before = rand(spans + 1, elements + 3)
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    slots = list(range(spans, 0, -1))
    want, want_state = torch.zeros(tokens, heads, vdim, device="cuda", dtype=torch.float64), before.double()
    share = heads // kv_heads
    q64, k64 = (x.double().view(tokens, kv_heads, dim).repeat_interleave(share, dim=1) for x in (q, k))
    v64, beta = v.double().view(tokens, heads, vdim), gates[:, :heads].double()
    for span, slot in enumerate(slots):
        s = want_state[slot, :elements].view(heads, dim, vdim).clone()
        for t in range(begins[span], begins[span + 1]):
            s = decay[t][:, None, None] * s
            u = beta[t][:, None] * (v64[t] - (s * k64[t].unsqueeze(-1)).sum(-2))
            s = s + k64[t].unsqueeze(-1) * u.unsqueeze(-2)
            want[t] = (s * q64[t].unsqueeze(-1)).sum(-2) * dim ** -0.5
        want_state[slot, :elements] = s.flatten()
    want = want.flatten(1)

    out, state = torch.zeros(tokens, heads * vdim, device="cuda"), before.clone()
    kernels.recurrent_scan(kernels.SCAN_DELTA, q, k, v, gates, out, state, state.stride(0), i32(begins), i32(slots), spans, heads,
                           kv_heads, dim, vdim, dim ** -0.5)
    chunks = tokens // 64 + spans
    full = lambda *shape: torch.full(shape, 5.0, device="cuda")                # noqa: E731
    plan, got, got_state, flag = torch.zeros(chunks + spans + 8, dtype=torch.int32, device="cuda"), full(tokens, heads * vdim), before.clone(), i32([0])
    kernels.chunk_plan(i32(begins), spans, chunks + 3, plan)
    operands = full(chunks * heads * kernels.delta_operand_bytes(dim) // 4)
    kernels.delta_chunk_scan(q, k, v, gates, pre_a, dt_bias, a_log, full(tokens, 2 * heads), full(tokens, heads), operands,
                             full(tokens, heads * vdim), full(chunks * elements), got, got_state, got_state.stride(0), i32(slots), plan,
                             chunks + 3, spans, chunks, heads, kv_heads, dim, vdim, dim ** -0.5, flag)
    assert int(flag.item()) == 0

    def off(x, y):
        return float((x.double() - y).norm() / y.norm())
    # float32 sums of the same products in different orders: errors of the same size, of a few units of 2^-24
    for name, a, b, c in (("read", got, out, want), ("state", got_state, state, want_state)):
        assert off(a, c) <= 2 * off(b, c) + 3e-7, (name, off(a, c), off(b, c))
    assert torch.equal(got_state[:, elements:], before[:, elements:]) and torch.equal(got_state[0], before[0])


@pytest.mark.parametrize("lengths,heads,dim,decay", [
    ([64, 65, 1, 128, 63], 3, 24, 0.0),              # whole chunks, one token more and less; a size between tiles
    ([300], 2, 64, -8.0),                            # almost nothing forgotten
    ([130, 66], 2, 7, 0.0),                          # odd columns: no access of two or four
    ([70, 200], 5, 64, 20.0),                        # every decay at its least: products of 1e-17 over a chunk
])
def test_generalised_delta_rule_in_chunks_of_64(lengths, heads, dim, decay):
    from celeg_b200 import kernels
    import math
    g = torch.Generator(device="cuda").manual_seed(13)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)      # noqa: E731
    tokens, spans, inner = sum(lengths), len(lengths), heads * dim
    proj, z = rand(tokens, 4 * inner + 4), rand(tokens, inner) + decay
    w0, a_bias, eps = rand(inner) * 0.3, rand(inner) * 0.3, 1e-6
    offsets = (0, inner, 2 * inner, 3 * inner)
    before = rand(spans + 1, inner * dim + 3)
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    slots = list(range(spans, 0, -1))
    r, k, v, a = (proj[:, o:o + inner].double().view(tokens, heads, dim) for o in offsets)
    keep = torch.exp(-math.exp(-0.5) * torch.sigmoid((z + w0).double())).view(tokens, heads, dim)
    unit = k / torch.sqrt(k.square().sum(-1, keepdim=True) + eps)
    removal = torch.sigmoid(a + a_bias.double().view(heads, dim)) * unit
    want, want_state = torch.zeros(tokens, heads, dim, device="cuda", dtype=torch.float64), before.double()
    for span, slot in enumerate(slots):
        s = want_state[slot, :inner * dim].view(heads, dim, dim).clone()
        for t in range(begins[span], begins[span + 1]):
            taken = (s * unit[t].unsqueeze(-1)).sum(-2)
            s = keep[t].unsqueeze(-1) * s - removal[t].unsqueeze(-1) * taken.unsqueeze(-2) + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
            want[t] = (s * r[t].unsqueeze(-1)).sum(-2)
        want_state[slot, :inner * dim] = s.flatten()
    want = want.flatten(1)

    token_span = i32([i for i, n in enumerate(lengths) for _ in range(n)])
    out, state, flag = torch.zeros(tokens, inner, device="cuda"), before.clone(), i32([0])
    records = torch.zeros(tokens * kernels.general_delta_scratch(heads, dim), device="cuda")
    kernels.general_delta_scan(proj, offsets, z, w0, a_bias, eps, token_span, i32(begins), i32(slots), records, out, state,
                               state.stride(0), tokens, spans, heads, dim, flag)
    chunks = tokens // 64 + spans
    full = lambda *shape: torch.full(shape, 5.0, device="cuda")                # noqa: E731
    plan, got, got_state = torch.zeros(chunks + spans + 8, dtype=torch.int32, device="cuda"), full(tokens, inner), before.clone()
    kernels.chunk_plan(i32(begins), spans, chunks + 3, plan)
    operands = full(chunks * heads * kernels.delta_operand_bytes(dim) // 4)
    kernels.general_delta_chunk_scan(proj, offsets, z, w0, a_bias, eps, full(tokens, inner), full(chunks * heads * 4096),
                                     full(chunks * heads * 4096), operands, full(tokens, inner), full(chunks * inner * dim),
                                     full(chunks * inner), got, got_state, got_state.stride(0), i32(slots), plan, chunks + 3, spans,
                                     chunks, heads, dim, flag)
    assert int(flag.item()) == 0

    def off(x, y):
        return float((x.double() - y).norm() / y.norm())
    # float32 sums of the same products in different orders: errors of the same size, of a few units of 2^-24
    for name, a, b, c in (("read", got, out, want), ("state", got_state, state, want_state)):
        assert off(a, c) <= 2 * off(b, c) + 3e-7, (name, off(a, c), off(b, c))
    assert torch.equal(got_state[:, inner * dim:], before[:, inner * dim:]) and torch.equal(got_state[0], before[0])
