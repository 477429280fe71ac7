"""The delta rule's decoding launch moves the carried inputs on itself (a key head's heads a cluster) or leaves them to a second
launch: each side of that rule, against the inputs moved by hand (exact: they are copies) and, after three tokens in turn, against the
steps that serve prompts."""
import pytest
import torch

from celeg_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,taps", [(4, 4, 64, 64, 4), (4, 2, 64, 64, 4), (8, 1, 32, 40, 2), (9, 1, 16, 24, 3),
                                                            (6, 2, 200, 300, 3), (3, 1, 40, 520, 16), (16, 2, 128, 128, 4),
                                                            (2, 1, 8, 8, 1)])
def test_carried_inputs_move_on(heads, kv_heads, dim, vdim, taps, tokens=3):
    torch.manual_seed(heads)
    qk, vw = kv_heads * dim, heads * vdim
    channels = 2 * qk + vw
    kernel = torch.randn(channels, taps, device="cuda") * 0.5
    a_log, dt_bias = torch.randn(heads, device="cuda") - 1.0, torch.randn(heads, device="cuda")
    norm = torch.rand(vdim, device="cuda") + 0.5
    elements = heads * dim * vdim
    stride = elements + (taps - 1) * channels + 4
    state = torch.randn(tokens, stride, device="cuda") * 0.3
    whole = state.clone()
    begins = torch.arange(tokens + 1, dtype=torch.int32, device="cuda")
    slots = (torch.arange(tokens, dtype=torch.int32, device="cuda") + 2) % tokens
    spans = torch.arange(tokens, dtype=torch.int32, device="cuda")
    gates, conv = torch.zeros(tokens, 2 * heads, device="cuda"), torch.zeros(tokens, channels, device="cuda")
    read, want, got = (torch.zeros(tokens, vw, device="cuda") for _ in range(3))
    for _ in range(3):
        proj = torch.randn(tokens, channels + vw + 2 * heads, device="cuda")
        before = whole[:, elements:elements + (taps - 1) * channels].clone().view(tokens, taps - 1, channels)
        kernels.recurrent_decode(kernels.SCAN_DELTA, proj, (0, qk, 2 * qk, channels, channels + vw, channels + vw + heads),
                                 kernel, whole[:, elements:], taps, channels, a_log, dt_bias, 0.0, norm, False, 1e-5,
                                 1e-6, whole, stride, begins, slots, tokens, heads, kv_heads, dim, vdim, dim ** -0.5, got)
        if taps > 1:
            moved = before.clone()
            moved[slots.long()] = torch.cat([before[slots.long()][:, 1:], proj[:, None, :channels]], dim=1)
            assert torch.equal(whole[:, elements:elements + (taps - 1) * channels].view(tokens, taps - 1, channels), moved)
        assert torch.equal(whole[:, -4:], state[:, -4:])
        kernels.delta_prepare(proj, kernel, state[:, elements:], stride, spans, begins, slots, conv,
                              proj[:, channels + vw:channels + vw + heads], proj[:, channels + vw + heads:], a_log, dt_bias,
                              gates, tokens, tokens, channels, taps, kv_heads, dim, heads, 1e-6)
        kernels.recurrent_scan(kernels.SCAN_DELTA, conv[:, :qk], conv[:, qk:2 * qk], conv[:, 2 * qk:], gates, read, state,
                               stride, begins, slots, tokens, heads, kv_heads, dim, vdim, dim ** -0.5)
        kernels.gated_head_norm(read, proj[:, channels:channels + vw], norm, False, want, tokens, heads, vdim, 1e-5,
                                kernels.GATE_SILU)
        # (the same formulas in float32 with sums in other orders over at most dim terms: a few times dim x 2^-24 of the largest)
        bound = 8 * dim * 2 ** -24
        assert float((got - want).abs().max()) <= bound * float(want.abs().max()) + 1e-5
        assert float((whole - state).abs().max()) <= bound * float(state.abs().max()) + 1e-5


@pytest.mark.parametrize("heads,kv_heads,most", [(4, 4, 74), (4, 2, 37), (8, 2, 16), (8, 1, 12)])
def test_carried_inputs_of_many_requests(heads, kv_heads, most):
    """The most requests whose launch moves the inputs on itself, and one more."""
    for tokens in (most, most + 1):
        assert kernels.decode_moves_carried(4, tokens, heads, kv_heads) == (tokens == most)
        test_carried_inputs_move_on(heads, kv_heads, 32, 40, 4, tokens)
