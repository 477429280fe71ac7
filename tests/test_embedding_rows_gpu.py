"""The gather of embedding rows on both sides of its rule: rows in eights and others, aligned buffers and others, against the
float32 product of the table's numbers. Each number is one product and (the copies) one rounding, so those are exact; a row's sum of
squares adds hidden terms in some order, whose rounding is at most hidden x 2^-24 of the sum."""
import pytest
import torch

from celeg_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden", [8, 100, 264, 2048, 2056, 5001])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(dtype, hidden, shift):
    torch.manual_seed(hidden)
    vocab, rows = 37, 5
    held = torch.randn(vocab * hidden + shift, device="cuda").to(dtype)
    table = held[shift:].view(vocab, hidden)
    tokens = torch.tensor([36, 0, 7, 7, 35], dtype=torch.int32, device="cuda")
    expected = table[tokens.long()].float() * 1.7
    out = torch.empty(rows, hidden, device="cuda")
    copy = torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16)
    kernels.embedding(table, tokens, out, 1.7, copy=copy)
    assert torch.equal(out, expected) and torch.equal(copy, expected.bfloat16())

    weight = torch.randn(hidden, device="cuda")
    first = kernels.SplitNorm(torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16),
                              torch.empty(rows, 1, device="cuda"), 1, 1e-5, hidden)
    out.zero_()
    kernels.embedding(table, tokens, out, 1.7, prepare=first, next_weight=weight)
    assert torch.equal(out, expected) and torch.equal(first.xw, (expected * weight).bfloat16())
    exact = expected.double().square().sum(1)
    assert bool(((first.sumsq[:, 0].double() - exact).abs() <= exact * hidden * 2 ** -24).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden", [64, 1000, 2048, 2056, 5000])
def test_squares_are_added_in_one_order(dtype, hidden):
    """A row's sum of squares has the same bits wherever the table and the outputs lie."""
    torch.manual_seed(hidden)
    vocab, rows = 11, 7
    tokens, weight = torch.randint(0, vocab, (rows,), dtype=torch.int32, device="cuda"), torch.randn(hidden, device="cuda")
    values = torch.randn(vocab, hidden, device="cuda").to(dtype)
    sums = []
    for shift in (0, 1):
        table = torch.empty(vocab * hidden + shift, device="cuda", dtype=dtype)[shift:].view(vocab, hidden)
        table.copy_(values)
        first = kernels.SplitNorm(torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16), torch.empty(rows, 1, device="cuda"), 1, 1e-5, hidden)
        kernels.embedding(table, tokens, torch.empty(rows, hidden, device="cuda"), 1.3, prepare=first, next_weight=weight)
        sums.append(first.sumsq.clone())
    assert torch.equal(*sums)
