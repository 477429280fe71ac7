"""Decode attention, a warp's tiles of 32 keys: contexts at the tiles' and the stages' ends, groups of query heads that fill half and
the whole of a 16-row tile, pages whose size is no power of two, maxima that grow late or never, against float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LENGTHS = [1, 31, 32, 33, 127, 128, 129, 256, 257, 640]


@pytest.mark.parametrize("chunk", [64, 256, 640])              # one stage a warp (chunks of at most 256), two
@pytest.mark.parametrize("heads,kv_heads,dim,page", [(8, 1, 64, 16), (9, 1, 64, 12), (16, 1, 128, 16), (4, 4, 64, 5), (6, 2, 96, 16),
                                                     (3, 1, 256, 7)])
def test_decode_attention_at_the_ends_of_tiles(heads, kv_heads, dim, page, chunk):
    from celeg_b200 import kernels
    rng = np.random.default_rng(heads + dim + chunk)
    tokens, group, scale = len(LENGTHS), heads // kv_heads, dim ** -0.5
    needs = [-(-n // page) for n in LENGTHS]
    order = rng.permutation(sum(needs)).tolist()
    table = np.full((tokens, max(needs)), -1, dtype=np.int32)
    bf16 = lambda x: torch.tensor(x, dtype=torch.float32).to(torch.bfloat16)                  # noqa: E731
    k = bf16(rng.normal(size=(sum(needs), kv_heads, page, dim)))
    v = bf16(rng.normal(size=(sum(needs), kv_heads, page, dim)))
    q = bf16(rng.normal(size=(tokens, heads, dim)))
    want = np.zeros((tokens, heads, dim))
    for t, n in enumerate(LENGTHS):
        table[t, :needs[t]] = [order.pop() for _ in range(needs[t])]
        pages = table[t, :needs[t]].tolist()
        if t % 3 == 1:                                          # scores that grow along the context: every tile has a new maximum
            for i, at in enumerate(pages):
                k[at] = bf16(np.float32(0.1 * i)) * q[t, ::group][:, None, :] / dim ** 0.5 + k[at] * 0.01
        if t % 3 == 2:                                          # ... or the first key stands out
            k[pages[0], :, 0] = q[t, ::group] * 2.0
        keys = k[pages].double().numpy().transpose(0, 2, 1, 3).reshape(-1, kv_heads, dim)[:n]
        values = v[pages].double().numpy().transpose(0, 2, 1, 3).reshape(-1, kv_heads, dim)[:n]
        for h in range(heads):
            s = keys[:, h // group] @ q[t, h].double().numpy() * scale
            w = np.exp(s - s.max())
            want[t, h] = (w / w.sum()) @ values[:, h // group]
    splits = -(-max(LENGTHS) // chunk)
    scratch = torch.empty(tokens * heads * splits * dim, device="cuda"), torch.empty(tokens * heads * splits * 2, device="cuda")
    counters, flag = torch.zeros(tokens * kv_heads, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros((tokens, heads * dim), dtype=torch.bfloat16, device="cuda")
    i32 = lambda x: torch.tensor(np.ascontiguousarray(x, dtype=np.int32), device="cuda")      # noqa: E731
    kernels.attention_decode(q.cuda().view(tokens, -1), heads * dim, out, k.cuda(), v.cuda(), i32([n - 1 for n in LENGTHS]),
                             i32(range(tokens)), i32(table), tokens, heads, kv_heads, dim, page, 0, scale, chunk, splits, *scratch,
                             counters, flag)
    assert int(flag.item()) == 0 and int(counters.abs().sum().item()) == 0
    # the weights are rounded to 8 bits before their product with values of order one, the output once more
    error = np.abs(out.double().cpu().numpy().reshape(tokens, heads, dim) - want)
    assert (error <= 2.0 ** -8 * (np.abs(want) + np.abs(v.double().numpy()).max() * 0.5)).all(), error.max()


@pytest.mark.parametrize("chunk", [256, 640])                  # one stage a warp, two
@pytest.mark.parametrize("heads,dim", [(1, 64), (16, 64), (4, 128)])
@pytest.mark.parametrize("n", [32, 160])                       # one warp's first tile, and its second
def test_weights_below_the_smallest_normal_number_count(n, heads, dim, chunk):
    """The first key's value is zero, the others' are 2^118 under weights of about 2^-130: bfloat16 holds such weights with three
    bits (2^-133), so an output is off by a sixteenth of itself at most, and by its own rounding."""
    from celeg_b200 import kernels
    page = 16
    pages = -(-n // page)
    k, v = torch.zeros((pages, 1, page, dim), dtype=torch.bfloat16), torch.full((pages, 1, page, dim), 2.0 ** 118, dtype=torch.bfloat16)
    k[..., 0], k[0, 0, 0, 0], v[0, 0, 0] = -90.0, 0.0, 0.0
    q = torch.zeros((1, heads, dim), dtype=torch.bfloat16)
    q[..., 0] = 1.0
    i32 = lambda x: torch.tensor(list(x), dtype=torch.int32, device="cuda")                   # noqa: E731
    splits = -(-n // chunk)
    scratch = torch.empty(heads * splits * dim, device="cuda"), torch.empty(heads * splits * 2, device="cuda")
    flag, out = i32([0]), torch.zeros((1, heads * dim), dtype=torch.bfloat16, device="cuda")
    kernels.attention_decode(q.cuda().view(1, -1), heads * dim, out, k.cuda(), v.cuda(), i32([n - 1]), i32([0]), i32(range(pages)).view(1, -1),
                             1, heads, 1, dim, page, 0, 1.0, chunk, splits, *scratch, i32([0]), flag)
    want = (n - 1) * np.exp(-90.0) * 2.0 ** 118
    assert int(flag.item()) == 0
    assert bool(((out.double() / want - 1.0).abs() <= 2.0 ** -4 + 2.0 ** -8).all()), float((out.double() / want).min())
