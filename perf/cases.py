"""What the speed of this package is measured on: its layers, each built from the part registry and run for one step as a
model runs it, and the engine's raw step over a whole (shallow) model.

A layer case is one mixer of one of the package's designs at the sizes that the designs have in bench.py (width 1,024 and
2,048, heads of 64 and 128), on normed activations of new requests. A pass zeroes the requests' state, as opening a request
does, and runs the mixer; it returns the mixer's output and the state (or the cache) that the pass left. An engine case is an
LFM2 model of four layers with LFM2-1.2B's widths behind Engine.forward."""
import hashlib
import json
import math
import os
import tempfile

import numpy as np
import torch

from celeg_b200 import Engine, EngineOptions, write_random_model
from celeg_b200.engine.step import StepEntry
from celeg_b200.parts import PagedBinding, Runtime, StateBinding, StepContext, part_factory

EPS = 1e-5
PAGE = 16
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def listed():
    return [
        # a server decoding for eight users: their prompts go in together, then twelve tokens each, logits of every step
        {"name": "engine_decode_b8", "kind": "engine", "width": 2048, "heads": 32, "kv_heads": 8, "requests": 8,
         "tokens": 512, "new": 12},
        # one long prompt through the whole model, the logits of its last token
        {"name": "engine_prompt", "kind": "engine", "width": 2048, "heads": 32, "kv_heads": 8, "requests": 1,
         "tokens": 2048, "new": 0},
        # the longest prompt, heads of 64 (LFM2, Ramosun, Liverax, Kodupel)
        layer("attention_prompt_64", "attention", 2048, 8192, 1, heads=32, kv_heads=8, dim=64),
        # two documents of unequal, odd lengths, heads of 128 (Naselorn, Fovezen)
        layer("attention_prompt_128", "attention", 2048, 4001, 2, heads=16, kv_heads=4, dim=128),
        # decoding with long contexts: what the cache's bytes cost
        layer("attention_decode_16k", "attention", 2048, 8, 8, heads=32, kv_heads=8, dim=64, context=16384),
        # Ramosun: the matrix memory with exponential gates, one prompt
        layer("mlstm_prompt", "mlstm", 2048, 2048, 1, heads=16, dim=64, vdim=128),
        # Ramosun: the gated delta rule, one prompt
        layer("gated_delta_prompt", "gated_delta", 2048, 2048, 1, heads=32, kv_heads=16, dim=64, vdim=64),
        # the smallest call: one token for each of two users
        layer("gated_delta_decode_b2", "gated_delta", 1024, 2, 2, heads=16, kv_heads=8, dim=64, vdim=64),
        # Kedesun: retention, three prompts of unequal lengths in one step
        layer("retention_prompt", "retention", 2048, 3001, 3, heads=16, dim=64, vdim=128),
        # Kodupel: the generalised delta rule with a decay a key channel, one prompt
        layer("general_delta_prompt", "general_delta", 2048, 2048, 1, heads=32, dim=64, vdim=64),
        # Fovezen: Mamba-2, one prompt
        layer("mamba2_prompt", "mamba2", 2048, 2048, 1, heads=64, kv_heads=8, dim=128, vdim=64),
        # Fovezen: gated linear attention, four prompts of unequal lengths in one step
        layer("linear_attention_prompt", "gated_linear_attention", 2048, 1999, 4, heads=16, dim=64, vdim=128),
    ]


def layer(name, kind, width, tokens, requests, heads, dim, vdim=0, kv_heads=0, context=0, dtype="bf16"):
    case = {"kind": kind, "width": width, "tokens": tokens, "requests": requests, "heads": heads, "kv_heads": kv_heads or heads,
            "dim": dim, "vdim": vdim or dim, "context": context, "dtype": dtype}
    return dict(case, name=name) if name else case


def draw(rng):
    kind = rng.choice(["attention", "attention", "mlstm", "gated_delta", "retention", "general_delta", "mamba2",
                       "gated_linear_attention"])
    width = rng.choice([768, 1024, 1536, 2048])
    if rng.random() < 0.25:                                     # decoding
        tokens = requests = rng.choice([1, 2, 3, 5, 8, 16, 24, 48])
        context = round(math.exp(rng.uniform(math.log(64), math.log(16384)))) if kind == "attention" else 0
        dtype = "bf16"
    else:
        dtype = "f32" if rng.random() < 0.1 else "bf16"
        tokens = round(math.exp(rng.uniform(math.log(200), math.log(500 if dtype == "f32" else 4096))))
        requests = rng.choice([1, 1, 2, 3, 6])
        context = 0
    if kind == "attention":
        dim = rng.choice([64, 64, 128, 128, 96, 256])
        heads = width // dim
        return layer("", kind, width, tokens, requests, heads, dim, kv_heads=rng.choice([n for n in (1, 2, 4, heads) if heads % n == 0]),
                     context=context, dtype=dtype)
    if kind == "mamba2":
        return layer("", kind, width, tokens, requests, width // 32, rng.choice([64, 128]), vdim=64, kv_heads=8, dtype=dtype)
    if kind == "general_delta":
        return layer("", kind, width, tokens, requests, width // 64, 64, dtype=dtype)
    if kind == "gated_delta":
        dim = rng.choice([64, 64, 32, 128])
        return layer("", kind, width, tokens, requests, width // 64, dim, vdim=rng.choice([64, 128]),
                     kv_heads=width // 64 // rng.choice([1, 2]), dtype=dtype)
    dim = rng.choice([64, 64, 32, 96, 128])
    return layer("", kind, width, tokens, requests, width // 128, dim, vdim=rng.choice([64, 128]), dtype=dtype)


# ------------------------------------------------------------------------------------------------ the step's requests
def lengths_of(case):
    """The tokens that each request brings: unequal, together ``tokens``."""
    n, tokens = case["requests"], case["tokens"]
    if tokens == n:
        return [1] * n
    shares = [2 + (5 * i) % 7 for i in range(n)]
    lengths = [max(2, tokens * s // sum(shares)) for s in shares]
    lengths[0] += tokens - sum(lengths)
    return lengths


def starts_of(case, lengths):
    """The positions that the requests' tokens begin at: a decoding request has a context behind it."""
    if not case["context"]:
        return [0] * len(lengths)
    return [max(0, case["context"] - 1 - 37 * i) for i in range(len(lengths))]


def generator_of(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(seed)


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def step_of(lengths, starts, table):
    begins = [0]
    for n in lengths:
        begins.append(begins[-1] + n)
    positions = [p for s, n in zip(starts, lengths) for p in range(s, s + n)]
    longest = max(s + n for s, n in zip(starts, lengths))
    bucket = 256
    while bucket < longest:
        bucket *= 2
    single = next((i for i, n in enumerate(lengths) if n != 1), len(lengths))
    return StepContext(tokens=begins[-1], spans=len(lengths), token_ids=i32([0] * begins[-1]), positions=i32(positions),
                       token_span=i32([i for i, n in enumerate(lengths) for _ in range(n)]), span_begin=i32(begins),
                       span_slot=i32(list(range(len(lengths)))), block_tables=[table] if table is not None else [],
                       error_flag=torch.zeros(1, dtype=torch.int32, device="cuda"), max_span=max(lengths), max_context=longest,
                       context_bucket=bucket, host_span_lengths=list(lengths), leading_single_tokens=single)


# -------------------------------------------------------------------------------------------------- weights and inputs
def weights_of(case, seed):
    """(params, weights as a checkpoint holds them: bfloat16 on the host). Matrices N(0, 1 / fan-in); steps, decays and gate
    biases as the methods' papers initialise them."""
    g = generator_of(seed)
    hidden, heads, kv, dim, vdim = (case[n] for n in ("width", "heads", "kv_heads", "dim", "vdim"))

    def matrix(rows, columns):
        return (torch.randn(rows, columns, device="cuda", generator=g) * columns ** -0.5).to(torch.bfloat16).cpu()

    def vector(n, mean=0.0, std=0.05):
        return (mean + std * torch.randn(n, device="cuda", generator=g)).to(torch.bfloat16).cpu()

    def spread(n, low, high):
        return (low + (high - low) * torch.rand(n, device="cuda", generator=g)).to(torch.bfloat16).cpu()

    def step_bias(n):                                           # softplus^-1 of a step between 0.001 and 0.1
        dt = torch.exp(math.log(1e-3) + (math.log(1e-1) - math.log(1e-3)) * torch.rand(n, device="cuda", generator=g))
        return (dt + torch.log(-torch.expm1(-dt))).to(torch.bfloat16).cpu()

    kind = case["kind"]
    params = {"hidden_size": hidden, "heads": heads, "dim": dim, "vdim": vdim, "eps": EPS}
    if kind == "attention":
        params = {"hidden_size": hidden, "num_heads": heads, "num_kv_heads": kv, "head_dim": dim, "qk_norm_eps": EPS,
                  "softmax_scale": dim ** -0.5}
        return params, {"q_proj": matrix(heads * dim, hidden), "k_proj": matrix(kv * dim, hidden), "v_proj": matrix(kv * dim, hidden),
                        "out_proj": matrix(hidden, heads * dim), "q_norm": vector(dim, 1.0), "k_norm": vector(dim, 1.0)}
    if kind == "mlstm":
        return dict(params, gate_cap=15.0), {
            "q": matrix(heads * dim, hidden), "k": matrix(heads * dim, hidden), "v": matrix(heads * vdim, hidden),
            "gate": matrix(heads * vdim, hidden), "input_gate": matrix(heads, hidden), "forget_gate": matrix(heads, hidden),
            "input_gate_bias": vector(heads, -2.0, 0.3), "forget_gate_bias": spread(heads, 3.0, 6.0),
            "norm": vector(heads * vdim, 1.0), "out": matrix(hidden, heads * vdim)}
    if kind == "gated_delta":
        return dict(params, kv_heads=kv, taps=4), {
            "q": matrix(kv * dim, hidden), "k": matrix(kv * dim, hidden), "v": matrix(heads * vdim, hidden),
            "gate": matrix(heads * vdim, hidden), "beta": matrix(heads, hidden), "decay": matrix(heads, hidden),
            "q_conv": matrix(kv * dim, 4), "k_conv": matrix(kv * dim, 4), "v_conv": matrix(heads * vdim, 4),
            "a_log": spread(heads, 0.0, math.log(16.0)), "dt_bias": step_bias(heads), "norm": vector(vdim, 1.0),
            "out": matrix(hidden, heads * vdim)}
    if kind == "retention":
        decay = [1.0 - 2.0 ** (-5.0 - 7.0 * h / max(heads - 1, 1)) for h in range(heads)]
        return dict(params, decay=decay), {
            "q": matrix(heads * dim, hidden), "k": matrix(heads * dim, hidden), "v": matrix(heads * vdim, hidden),
            "gate": matrix(heads * vdim, hidden), "out": matrix(hidden, heads * vdim)}
    rank = max(hidden // 32, 8)
    if kind == "general_delta":
        inner = heads * dim
        names = {n: matrix(inner, hidden) for n in ("r", "k", "v", "gate", "removal")}
        return params, dict(names, decay_down=matrix(rank, hidden), decay_up=matrix(inner, rank), removal_bias=vector(inner),
                            decay_bias=vector(inner, 0.0, 0.3), norm=vector(inner, 1.0), out=matrix(hidden, inner))
    if kind == "mamba2":
        inner, shared = heads * vdim, kv * dim
        return {"hidden_size": hidden, "heads": heads, "vdim": vdim, "state": dim, "groups": kv, "taps": 4, "norm_groups": kv,
                "eps": EPS}, {
            "in_proj": matrix(2 * inner + 2 * shared + heads, hidden), "conv": matrix(inner + 2 * shared, 4),
            "conv_bias": vector(inner + 2 * shared), "dt_bias": step_bias(heads), "a_log": spread(heads, 0.0, math.log(16.0)),
            "direct": vector(heads, 1.0), "norm": vector(inner, 1.0), "out": matrix(hidden, inner)}
    if kind == "gated_linear_attention":
        return dict(params, tau=16.0), {
            "q": matrix(heads * dim, hidden), "k": matrix(heads * dim, hidden), "v": matrix(heads * vdim, hidden),
            "gate": matrix(heads * vdim, hidden), "decay_down": matrix(rank, hidden), "decay_up": matrix(heads * dim, rank),
            "decay_bias": vector(heads * dim), "norm": vector(vdim, 1.0), "out": matrix(hidden, heads * vdim)}
    raise ValueError(kind)


def activations_of(case, seed):
    """Normed activations: order one, bfloat16 (so both precisions get the same values)."""
    return torch.randn(case["tokens"], case["width"], device="cuda", generator=generator_of(seed + 7919)).to(torch.bfloat16)


def cache_of(case, seed):
    """(lengths, starts, page table, keys, values): normed keys and values of order one at the positions that were there."""
    lengths = lengths_of(case)
    starts = starts_of(case, lengths)
    needs = [-(-(s + n) // PAGE) for s, n in zip(starts, lengths)]
    host = generator_of(seed + 31, "cpu")
    order = torch.randperm(sum(needs), generator=host).tolist()  # a request's pages lie anywhere
    table = np.full((len(lengths), max(needs)), -1, dtype=np.int32)
    for i, need in enumerate(needs):
        table[i, :need] = [order.pop() for _ in range(need)]
    shape = (sum(needs), case["kv_heads"], PAGE, case["dim"])
    if not case["context"]:
        return lengths, starts, table, torch.zeros(shape, device="cuda"), torch.zeros(shape, device="cuda")
    g = generator_of(seed + 63)
    return (lengths, starts, table, torch.randn(shape, device="cuda", generator=g).to(torch.bfloat16),
            torch.randn(shape, device="cuda", generator=g).to(torch.bfloat16))


# ------------------------------------------------------------------------------------------------------------- passes
def lfm2_config(case):
    types = ["conv", "full_attention", "conv", "full_attention"]
    return {"model_type": "lfm2", "vocab_size": 16384, "hidden_size": case["width"], "num_hidden_layers": len(types),
            "num_attention_heads": case["heads"], "num_key_value_heads": case["kv_heads"], "head_dim": 64,
            "intermediate_size": 4 * case["width"], "conv_L_cache": 3, "rope_theta": 1000000.0, "norm_eps": EPS,
            "tie_word_embeddings": True, "max_position_embeddings": 4096, "layer_types": types, "bos_token_id": 1,
            "eos_token_id": 7, "pad_token_id": 0}


def folder_of(raw):
    """A model folder with random weights, written once."""
    tag = hashlib.sha256(json.dumps(raw, sort_keys=True).encode()).hexdigest()[:16]
    folder = os.path.join(tempfile.gettempdir(), f"celeg_b200_cases_{os.getuid()}_{tag}")
    if not os.path.isfile(os.path.join(folder, "complete")):
        write_random_model(folder, raw, 0)
        with open(os.path.join(folder, "complete"), "w") as handle:
            handle.write("ok")
    return folder


def token_ids(case, raw, seed):
    """Per request its prompt and the tokens fed after it."""
    each = case["tokens"] // case["requests"]
    host = generator_of(seed, "cpu")
    return [torch.randint(0, raw["vocab_size"], (each + case["new"],), generator=host).tolist() for _ in range(case["requests"])]


def prepare(case, seed):
    if case["kind"] == "engine":
        raw = lfm2_config(case)
        each = case["tokens"] // case["requests"]
        options = EngineOptions(max_active_requests=case["requests"], max_batched_tokens=case["tokens"],
                                prefill_chunk_tokens=case["tokens"], page_tokens=PAGE,
                                logical_kv_pages=case["requests"] * (-(-(each + case["new"]) // PAGE)))
        engine = Engine(folder_of(raw), max_context=each + case["new"], options=options)
        return {"case": case, "engine": engine, "tokens": token_ids(case, raw, seed), "each": each}
    dtype = DTYPES[case["dtype"]]
    params, weights = weights_of(case, seed)
    lengths = lengths_of(case)
    longest = max(s + n for s, n in zip(starts_of(case, lengths), lengths))
    rows = -(-case["tokens"] // 64) * 64
    rt = Runtime(torch.device("cuda:0"), dtype, rows, max_requests=max(8, case["requests"]), max_context=max(4096, longest))
    x = torch.zeros((rows, case["width"]), dtype=dtype, device="cuda")
    x[:case["tokens"]] = activations_of(case, seed).to(dtype)
    state = {"case": case, "x": x, "out": torch.zeros_like(x), "rt": rt}
    if case["kind"] == "attention":
        rope = part_factory("position", "rope_split_half")({"theta": 1000000.0, "head_dim": case["dim"], "rotary_dim": case["dim"]}, rt)
        state["mixer"] = part_factory("mixer", "attention")(params, weights, {"position": rope}, rt)
        lengths, starts, table, k, v = cache_of(case, seed)
        state["cache"] = (k.to(dtype), v.to(dtype))
        state["mixer"].bind_cache(PagedBinding(group=0, k=state["cache"][0], v=state["cache"][1], page_tokens=PAGE))
        state["step"] = step_of(lengths, starts, i32(table))
    else:
        state["mixer"] = part_factory("mixer", case["kind"])(params, weights, {}, rt)
        elements = state["mixer"].cache_need().elements
        state["slots"] = torch.zeros((case["requests"], -(-elements // 4) * 4), dtype=torch.float32, device="cuda")
        state["mixer"].bind_cache(StateBinding(state=state["slots"], slot_stride=state["slots"].stride(0)))
        state["step"] = step_of(lengths, [0] * len(lengths), None)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "engine":
        return run_engine(state)
    step, tokens = state["step"], case["tokens"]
    step.extras.clear()
    if "slots" in state:
        state["slots"].zero_()                                  # new requests
    state["mixer"].forward(state["x"], state["out"], step)
    if "slots" in state:
        return state["out"][:tokens], state["slots"]
    if case["context"]:
        return (state["out"][:tokens],)
    return state["out"][:tokens], state["cache"]


def run_engine(state):
    case, engine, tokens, each = state["case"], state["engine"], state["tokens"], state["each"]
    ids = list(range(case["requests"]))
    logits = [engine.forward([StepEntry(i, tokens[i][:each], [each - 1]) for i in ids]).clone()]
    for at in range(each, each + case["new"]):
        logits.append(engine.forward([StepEntry(i, [tokens[i][at]], [0]) for i in ids]).clone())
    for i in ids:
        engine.end(i)
    return logits


# ------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    h, t = case["width"], case["tokens"]
    if case["kind"] == "engine":
        q, kv, inner, vocab = case["heads"] * 64, case["kv_heads"] * 64, 4 * case["width"], 16384
        weights = 2 * 4 * h * h + 2 * ((q + 2 * kv) * h + q * h) + 4 * 3 * h * inner
        rows = case["requests"] * (1 + case["new"])
        each = t // case["requests"]
        scores = case["requests"] * 2 * 2 * 2 * q * (each + case["new"]) ** 2 / 2
        steps = 1 + case["new"]
        return {"bytes": steps * 2.0 * (weights + vocab * h) + 4.0 * rows * vocab,
                "flops": 2.0 * (t + case["requests"] * case["new"]) * weights + 2.0 * rows * vocab * h + scores}
    heads, kv, dim, vdim = (case[n] for n in ("heads", "kv_heads", "dim", "vdim"))
    size = 4 if case["dtype"] == "f32" else 2
    lengths = lengths_of(case)
    starts = starts_of(case, lengths)
    rank = max(h // 32, 8)
    inner = {"attention": heads * dim}.get(case["kind"], heads * vdim)
    columns = {"attention": (heads + 2 * kv) * dim, "mlstm": 2 * heads * (dim + vdim) + 2 * heads,
               "gated_delta": 2 * kv * dim + 2 * heads * vdim + 2 * heads, "retention": 2 * heads * (dim + vdim),
               "general_delta": 5 * heads * dim + rank + rank * heads * dim // h,
               "mamba2": 2 * heads * vdim + 2 * kv * dim + heads,
               "gated_linear_attention": 2 * heads * (dim + vdim) + rank + rank * heads * dim // h}[case["kind"]]
    flops = 2.0 * t * h * (columns + inner)
    moved = size * (h * (columns + inner) + 2.0 * t * h)
    if case["kind"] == "attention":
        seen = sum(n * s + n * (n + 1) / 2 for s, n in zip(starts, lengths))
        flops += 4.0 * heads * dim * seen
        moved += size * 2.0 * kv * dim * sum(s + n for s, n in zip(starts, lengths))
    else:
        flops += (6.0 if "delta" in case["kind"] else 4.0) * t * heads * dim * vdim
        moved += 2 * 4.0 * case["requests"] * heads * dim * vdim
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """bfloat16: q, k, attention outputs and gated read-outs are rounded to 8 bits between the products, and the result is;
    float32: sums of about two thousand terms in any order, through unit norms and root mean squares."""
    if case["kind"] == "engine":
        return {"rel": 3e-2, "max": 0.2}           # four layers: a rounding of the first travels through the others
    return {"rel": 2e-5, "max": 2e-3} if case["dtype"] == "f32" else {"rel": 1e-2, "max": 0.1}


# ---------------------------------------------------------------------------------------------------- 64-bit results
def exact(case, seed):
    if case["kind"] == "engine":
        return exact_engine(case, seed)
    params, weights = weights_of(case, seed)
    w = {name: tensor.double().cuda() for name, tensor in weights.items()}
    x = activations_of(case, seed).double()
    if case["kind"] == "attention":
        return exact_attention(case, seed, w, x)
    lengths = lengths_of(case)
    read, state = RECURRENCES[case["kind"]](case, params, w, x, lengths)
    pad = -state.shape[1] % 4
    return read @ w["out"].T, torch.cat([state, torch.zeros(len(lengths), pad, device="cuda", dtype=torch.float64)], dim=1)


def rms(x):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS)


def rope(x, positions):
    """Pairs (i, i + half) of the last axis; x [tokens, heads, dim]."""
    half = x.shape[-1] // 2
    frequency = torch.pow(torch.tensor(1000000.0, dtype=torch.float64), torch.arange(half, dtype=torch.float64) / -half)
    angle = positions.double()[:, None, None] * frequency.float().double().cuda()
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def attend(q, k, v, first):
    """q [n, heads, d] at positions first.., k, v [m, kv, d]; causal."""
    group = q.shape[1] // k.shape[1]
    hidden = torch.arange(k.shape[0], device="cuda")[None] > (first + torch.arange(q.shape[0], device="cuda"))[:, None]
    out = torch.empty_like(q)
    for h in range(q.shape[1]):
        scores = (q[:, h] @ k[:, h // group].T) * q.shape[-1] ** -0.5
        out[:, h] = torch.softmax(scores.masked_fill_(hidden, -math.inf), dim=-1) @ v[:, h // group]
    return out


def exact_attention(case, seed, w, x):
    heads, kv, dim = case["heads"], case["kv_heads"], case["dim"]
    lengths, starts, table, k_pages, v_pages = cache_of(case, seed)
    k_pages, v_pages = k_pages.double(), v_pages.double()
    rows, at = [], 0
    for i, (start, n) in enumerate(zip(starts, lengths)):
        part = x[at:at + n]
        at += n
        positions = torch.arange(start, start + n, device="cuda")
        q = rope(rms((part @ w["q_proj"].T).view(n, heads, dim)) * w["q_norm"], positions)
        k = rope(rms((part @ w["k_proj"].T).view(n, kv, dim)) * w["k_norm"], positions)
        v = (part @ w["v_proj"].T).view(n, kv, dim)
        pages = torch.tensor(table[i], device="cuda", dtype=torch.long)
        page, slot = pages[positions // PAGE], positions % PAGE
        k_pages[page, :, slot] = k
        v_pages[page, :, slot] = v
        mine = pages[pages >= 0]
        all_k = k_pages[mine].permute(0, 2, 1, 3).reshape(-1, kv, dim)[:start + n]
        all_v = v_pages[mine].permute(0, 2, 1, 3).reshape(-1, kv, dim)[:start + n]
        rows.append(attend(q, all_k, all_v, start).reshape(n, heads * dim))
    out = torch.cat(rows) @ w["out_proj"].T
    return (out,) if case["context"] else (out, (k_pages, v_pages))


def by_request(lengths, *tensors):
    """Every tensor [tokens, ...] as [longest, requests, ...] (zeros past a request's end), and whether a place is a token."""
    at, longest = 0, max(lengths)
    real = torch.zeros((longest, len(lengths)), device="cuda", dtype=torch.bool)
    padded = [torch.zeros((longest, len(lengths), *t.shape[1:]), device="cuda", dtype=torch.float64) for t in tensors]
    for i, n in enumerate(lengths):
        for p, t in zip(padded, tensors):
            p[:n, i] = t[at:at + n]
        real[:n, i] = True
        at += n
    return real, padded


def gather_back(lengths, padded):
    return torch.cat([padded[:n, i] for i, n in enumerate(lengths)])


def convolved(x, kernel, bias, lengths):
    """Causal taps per channel and SiLU, and the last taps - 1 inputs of each request [requests, taps - 1, channels]."""
    taps, out, last, at = kernel.shape[1], [], [], 0
    for n in lengths:
        rows = torch.cat([torch.zeros(taps - 1, x.shape[1], device="cuda", dtype=torch.float64), x[at:at + n]])
        total = sum(kernel[:, j] * rows[j:j + n] for j in range(taps)) + (bias if bias is not None else 0.0)
        out.append(torch.nn.functional.silu(total))
        last.append(rows[n:])
        at += n
    return torch.cat(out), torch.stack(last)


def linear_scan(lengths, q, k, v, decay):
    """S' = diag(decay) S + k v^T, S'^T q; q, k [t, heads, dim], v [t, heads, vdim], decay [t, heads, dim or 1]."""
    real, (q, k, v, decay) = by_request(lengths, q, k, v, decay)
    s = torch.zeros((*q.shape[1:], v.shape[-1]), device="cuda", dtype=torch.float64)
    outs = torch.zeros_like(v)
    for t in range(q.shape[0]):
        new = decay[t].unsqueeze(-1) * s + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
        s = torch.where(real[t][:, None, None, None], new, s)
        outs[t] = (s * q[t].unsqueeze(-1)).sum(-2)
    return gather_back(lengths, outs), s.flatten(1)


def exact_retention(case, params, w, x, lengths):
    heads, dim, vdim, n = case["heads"], case["dim"], case["vdim"], case["tokens"]
    q, k = (x @ w["q"].T).view(n, heads, dim), (x @ w["k"].T).view(n, heads, dim) * dim ** -0.5
    v, gate = (x @ w["v"].T).view(n, heads, vdim), (x @ w["gate"].T).view(n, heads, vdim)
    decay = torch.tensor(params["decay"], dtype=torch.float32).double().cuda().view(1, heads, 1).expand(n, heads, 1)
    read, state = linear_scan(lengths, q, k, v, decay)
    return (rms(read) * torch.nn.functional.silu(gate)).flatten(1), state


def exact_linear_attention(case, params, w, x, lengths):
    heads, dim, vdim, n = case["heads"], case["dim"], case["vdim"], case["tokens"]
    q, k = (x @ w["q"].T).view(n, heads, dim) * dim ** -0.5, (x @ w["k"].T).view(n, heads, dim)
    v, gate = (x @ w["v"].T).view(n, heads, vdim), (x @ w["gate"].T).view(n, heads, vdim)
    z = x @ w["decay_down"].T @ w["decay_up"].T + w["decay_bias"]
    decay = torch.exp(torch.nn.functional.logsigmoid(z) / params["tau"]).view(n, heads, dim)
    read, state = linear_scan(lengths, q, k, v, decay)
    return (rms(read) * w["norm"] * torch.nn.functional.silu(gate)).flatten(1), state


def exact_mamba2(case, params, w, x, lengths):
    heads, groups, dim, vdim, n = case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["tokens"]
    inner, shared = heads * vdim, groups * dim
    rows = x @ w["in_proj"].T
    z, mixed, raw = rows[:, :inner], rows[:, inner:2 * inner + 2 * shared], rows[:, 2 * inner + 2 * shared:]
    mixed, carried = convolved(mixed, w["conv"], w["conv_bias"], lengths)
    v = mixed[:, :inner].view(n, heads, vdim)
    k = mixed[:, inner:inner + shared].view(n, groups, dim).repeat_interleave(heads // groups, dim=1)
    q = mixed[:, inner + shared:].view(n, groups, dim).repeat_interleave(heads // groups, dim=1)
    dt = torch.nn.functional.softplus(raw + w["dt_bias"], threshold=100.0)
    read, state = linear_scan(lengths, q, k * dt.unsqueeze(-1), v, torch.exp(-torch.exp(w["a_log"]) * dt).unsqueeze(-1))
    read = (read + w["direct"][:, None] * v).flatten(1) * torch.nn.functional.silu(z)
    read = rms(read.view(n, params["norm_groups"], -1)).flatten(1) * w["norm"]
    return read, torch.cat([state, carried.flatten(1)], dim=1)


def exact_mlstm(case, params, w, x, lengths):
    heads, dim, vdim, n = case["heads"], case["dim"], case["vdim"], case["tokens"]
    cap = params["gate_cap"]
    q, k = (x @ w["q"].T).view(n, heads, dim) * dim ** -0.5, (x @ w["k"].T).view(n, heads, dim)
    v, gate = (x @ w["v"].T).view(n, heads, vdim), (x @ w["gate"].T).view(n, heads, vdim)
    i = cap * torch.tanh((x @ w["input_gate"].T + w["input_gate_bias"]) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((x @ w["forget_gate"].T + w["forget_gate_bias"]) / cap))
    real, (q, k, v, i, f) = by_request(lengths, q, k, v, i, f)
    s = torch.zeros((*q.shape[1:], vdim), device="cuda", dtype=torch.float64)
    norm, m = torch.zeros(q.shape[1:], device="cuda", dtype=torch.float64), torch.zeros(q.shape[1:3], device="cuda", dtype=torch.float64)
    outs = torch.zeros_like(v)
    for t in range(q.shape[0]):
        peak = torch.maximum(f[t] + m, i[t])
        keep, write = torch.exp(f[t] + m - peak), torch.exp(i[t] - peak)
        there = real[t][:, None]
        s = torch.where(there[..., None, None], keep[..., None, None] * s + (write[..., None] * k[t]).unsqueeze(-1) * v[t].unsqueeze(-2), s)
        norm = torch.where(there[..., None], keep[..., None] * norm + write[..., None] * k[t], norm)
        m = torch.where(there, peak, m)
        lower = torch.maximum((norm * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        outs[t] = (s * q[t].unsqueeze(-1)).sum(-2) / lower[..., None]
    read = rms(gather_back(lengths, outs)).flatten(1) * w["norm"] * torch.sigmoid(gate.flatten(1))
    return read, torch.cat([s.flatten(1), norm.flatten(1), m], dim=1)


def exact_gated_delta(case, params, w, x, lengths):
    heads, kv, dim, vdim, n = case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["tokens"]
    mixed, carried = convolved(torch.cat([x @ w["q"].T, x @ w["k"].T, x @ w["v"].T], dim=1),
                               torch.cat([w["q_conv"], w["k_conv"], w["v_conv"]]), None, lengths)
    q, k = mixed[:, :kv * dim].view(n, kv, dim), mixed[:, kv * dim:2 * kv * dim].view(n, kv, dim)
    v, gate = mixed[:, 2 * kv * dim:].view(n, heads, vdim), (x @ w["gate"].T).view(n, heads, vdim)
    q = (q / torch.sqrt(q.square().sum(-1, keepdim=True) + 1e-6) * dim ** -0.5).repeat_interleave(heads // kv, dim=1)
    k = (k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(heads // kv, dim=1)
    beta = torch.sigmoid(x @ w["beta"].T)
    decay = torch.exp(-torch.exp(w["a_log"]) * torch.nn.functional.softplus(x @ w["decay"].T + w["dt_bias"], threshold=100.0))
    real, (q, k, v, beta, decay) = by_request(lengths, q, k, v, beta, decay)
    s = torch.zeros((*q.shape[1:], vdim), device="cuda", dtype=torch.float64)
    outs = torch.zeros_like(v)
    for t in range(q.shape[0]):
        kept = decay[t][..., None, None] * s
        u = beta[t][..., None] * (v[t] - (kept * k[t].unsqueeze(-1)).sum(-2))
        s = torch.where(real[t][:, None, None, None], kept + k[t].unsqueeze(-1) * u.unsqueeze(-2), s)
        outs[t] = (s * q[t].unsqueeze(-1)).sum(-2)
    read = (rms(gather_back(lengths, outs)) * w["norm"] * torch.nn.functional.silu(gate)).flatten(1)
    return read, torch.cat([s.flatten(1), carried.flatten(1)], dim=1)


def exact_general_delta(case, params, w, x, lengths):
    heads, dim, n = case["heads"], case["dim"], case["tokens"]
    r, k, v, gate = ((x @ w[name].T).view(n, heads, dim) for name in ("r", "k", "v", "gate"))
    keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ w["decay_down"].T) @ w["decay_up"].T + w["decay_bias"]))
    removal = torch.sigmoid(x @ w["removal"].T + w["removal_bias"]).view(n, heads, dim)
    unit = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    real, (r, k, v, keep, removal, unit) = by_request(lengths, r, k, v, keep.view(n, heads, dim), removal, unit)
    s = torch.zeros((*r.shape[1:], dim), device="cuda", dtype=torch.float64)
    outs = torch.zeros_like(v)
    for t in range(r.shape[0]):
        taken = (s * unit[t].unsqueeze(-1)).sum(-2)
        new = keep[t].unsqueeze(-1) * s - (removal[t] * unit[t]).unsqueeze(-1) * taken.unsqueeze(-2) + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
        s = torch.where(real[t][:, None, None, None], new, s)
        outs[t] = (s * r[t].unsqueeze(-1)).sum(-2)
    return rms(gather_back(lengths, outs)).flatten(1) * w["norm"] * torch.sigmoid(gate.flatten(1)), s.flatten(1)


RECURRENCES = {"retention": exact_retention, "gated_linear_attention": exact_linear_attention, "mamba2": exact_mamba2,
               "mlstm": exact_mlstm, "gated_delta": exact_gated_delta, "general_delta": exact_general_delta}


def exact_engine(case, seed):
    from celeg_b200.weights import SafetensorsFile
    raw = lfm2_config(case)
    stored = SafetensorsFile(os.path.join(folder_of(raw), "model.safetensors"))
    w = lambda name: stored.tensor(name).double().cuda()        # noqa: E731
    each, heads, kv = case["tokens"] // case["requests"], case["heads"], case["kv_heads"]
    table = w("model.embed_tokens.weight")
    outs = [[] for _ in range(1 + case["new"])]
    norm = lambda x, name: rms(x) * w(name)                     # noqa: E731
    for ids in token_ids(case, raw, seed):
        x = table[torch.tensor(ids, device="cuda")]
        n = len(ids)
        positions = torch.arange(n, device="cuda")
        for i, kind in enumerate(raw["layer_types"]):
            at = f"model.layers.{i}."
            y = norm(x, at + "operator_norm.weight")
            if kind == "conv":
                b, c, g = (y @ w(at + "conv.in_proj.weight").T).chunk(3, dim=-1)
                taps = w(at + "conv.conv.weight").reshape(-1, 3)
                rows = torch.cat([torch.zeros(2, x.shape[1], device="cuda", dtype=torch.float64), b * g])
                y = (c * sum(taps[:, j] * rows[j:j + n] for j in range(3))) @ w(at + "conv.out_proj.weight").T
            else:
                a = at + "self_attn."
                q = rope(norm((y @ w(a + "q_proj.weight").T).view(n, heads, 64), a + "q_layernorm.weight"), positions)
                k = rope(norm((y @ w(a + "k_proj.weight").T).view(n, kv, 64), a + "k_layernorm.weight"), positions)
                v = (y @ w(a + "v_proj.weight").T).view(n, kv, 64)
                y = attend(q, k, v, 0).reshape(n, -1) @ w(a + "out_proj.weight").T
            x = x + y
            y = norm(x, at + "ffn_norm.weight")
            gate, up = y @ w(at + "feed_forward.w1.weight").T, y @ w(at + "feed_forward.w3.weight").T
            x = x + (torch.nn.functional.silu(gate) * up) @ w(at + "feed_forward.w2.weight").T
        rows = norm(x[each - 1:], "model.embedding_norm.weight") @ table.T
        for j in range(1 + case["new"]):
            outs[j].append(rows[j])
    return [torch.stack(rows) for rows in outs]
