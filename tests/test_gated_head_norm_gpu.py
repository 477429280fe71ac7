"""The gated norm of heads of 16 to 128 entries, four neighbours a lane, against 64 bits: ends of blocks, shared and own weights,
both orders of gate and norm, and rows whose gates do not start on 16 bytes (which take two neighbours or one a lane)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float32, torch.bfloat16))
@pytest.mark.parametrize("offset", (0, 4, 2, 1))
@pytest.mark.parametrize("vdim,tokens,heads", ((16, 1, 1), (16, 11, 3), (32, 17, 5), (64, 9, 1), (64, 33, 7), (128, 5, 1), (128, 3, 3)))
def test_heads_of_powers_of_two(vdim, tokens, heads, offset, dtype):
    from celeg_b200 import kernels
    torch.manual_seed(vdim + tokens)
    width, eps = heads * vdim, 1e-5
    o = torch.randn(tokens, width, device="cuda") * 4.0
    rows = torch.randn(tokens, width + 8, device="cuda") * 3.0
    gate = rows[:, offset:offset + width]
    shared = 1.0 + 0.2 * torch.randn(vdim, device="cuda")
    own = 1.0 + 0.2 * torch.randn(width, device="cuda")
    for weight, per_head in ((None, False), (shared, False), (own, True)):
        for kind in (kernels.GATE_SIGMOID, kernels.GATE_SILU):
            for before in (0, kernels.GATE_BEFORE_NORM):
                out = torch.full((tokens + 1, width), 7.0, dtype=dtype, device="cuda")
                kernels.gated_head_norm(o, gate, weight, per_head, out, tokens, heads, vdim, eps, kind + before)
                g = torch.sigmoid(gate.double())
                z = (g * gate.double() if kind == kernels.GATE_SILU else g).reshape(tokens, heads, vdim)
                x = o.double().reshape(tokens, heads, vdim)
                if before:
                    x = x * z
                y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
                if weight is not None:
                    y = y * weight.double().reshape(heads if per_head else 1, vdim)
                want = (y if before else y * z).reshape(tokens, width)
                # a gate of up to 8 roundings (an exponential of 2, a sum, a quotient of 2, a product), twice where the sum of
                # squares holds it as well; log2(vdim) + 3 for the mean, halved by the root; 6 for the products and the quotient
                bound = 32 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
                assert ((out[:tokens].double() - want).abs() <= bound * want.abs() + 1e-30).all()
                assert (out[tokens] == 7.0).all()
