"""Short convolutions over portions, a thread several tokens: spans that begin anywhere in a tile, tiles with fewer tokens, every
head size of the delta rule's preparation that has a kernel of tiles, against float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(x):
    return torch.tensor(x, device="cuda")


def convolved(proj, kernel, carried, lengths, slots):
    """float64 sums of the taps [tokens, channels] and the inputs carried on, per slot [taps - 1, channels]."""
    taps = kernel.shape[1]
    out, carry, at = [], {}, 0
    for length, slot in zip(lengths, slots):
        rows = np.concatenate([carried[slot], proj[at:at + length]]).astype(np.float64)
        out.append(sum(rows[j:j + length] * kernel[:, j] for j in range(taps)))
        carry[slot] = rows[length:]
        at += length
    return np.concatenate(out), carry


def silu(x):
    return x / (1.0 + np.exp(-x))


def spans_of(lengths):
    begins = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    return dev(np.repeat(np.arange(len(lengths)), lengths).astype(np.int32)), dev(begins)


LENGTHS = [[63], [64], [61, 1, 2, 3, 1, 9], [1, 1, 1, 70], [7, 8, 9, 40, 17], [200]]


# Tiles from 741 tokens on, with 4,132 channels from 64: the last step without them and the first with; spans of 1 to 3 tokens begin
# inside tiles, and a block along the channels may have few of them
@pytest.mark.parametrize("lengths", LENGTHS + [[740], [741], [725, 1, 2, 3, 1, 9], [1, 1, 1, 740]])
@pytest.mark.parametrize("dim,kv_heads,vw", [(32, 3, 100), (64, 2, 64), (128, 5, 36), (128, 16, 36)])
def test_delta_prepare_in_tiles(lengths, dim, kv_heads, vw):
    from celeg_b200 import kernels
    rng = np.random.default_rng(len(lengths) + dim)
    tokens, heads, qk = sum(lengths), 2 * kv_heads, kv_heads * dim
    channels, gates_at = 2 * qk + vw, 2 * qk + vw
    stride = (channels + 2 * heads + 3) // 4 * 4
    proj = rng.normal(size=(tokens, stride)).astype(np.float32)
    kernel = rng.normal(size=(channels, 4)).astype(np.float32)
    slots = list(rng.permutation(len(lengths)))
    carried = rng.normal(size=(len(lengths), 3, channels)).astype(np.float32)
    a_log, dt_bias = rng.normal(size=heads).astype(np.float32), rng.normal(size=heads).astype(np.float32)
    state = torch.zeros((len(lengths), 3 * channels + 4), device="cuda")
    state[:, :3 * channels] = dev(carried.reshape(len(lengths), -1))
    span, begins = spans_of(lengths)
    proj_dev, conv = dev(proj), torch.zeros((tokens, channels), device="cuda")
    gates = torch.zeros((tokens, 2 * heads), device="cuda")
    kernels.delta_prepare(proj_dev, dev(kernel), state, state.stride(0), span, begins, dev(np.array(slots, dtype=np.int32)), conv,
                          proj_dev[:, gates_at:], proj_dev[:, gates_at + heads:], dev(a_log), dev(dt_bias), gates, tokens,
                          len(lengths), channels, 4, kv_heads, dim, heads, 1e-6)
    sums, carry = convolved(proj[:, :channels], kernel, carried, lengths, slots)
    want = silu(sums)
    units = want[:, :2 * qk].reshape(tokens, 2 * kv_heads, dim)
    units /= np.sqrt((units * units).sum(-1, keepdims=True) + 1e-6)
    # a sum of four products of order one, SiLU and a unit norm: ten roundings of 2^-24 of the largest product
    assert np.abs(conv.cpu().numpy() - want).max() < 10 * 2.0 ** -24 * max(1.0, np.abs(sums).max())
    beta = 1.0 / (1.0 + np.exp(-proj[:, gates_at:gates_at + heads].astype(np.float64)))
    decay = np.exp(-np.exp(a_log.astype(np.float64)) * np.log1p(np.exp(proj[:, gates_at + heads:gates_at + 2 * heads].astype(np.float64) + dt_bias)))
    assert np.abs(gates.cpu().numpy() - np.concatenate([beta, decay], axis=1)).max() < 2e-6
    for slot, rows in carry.items():
        assert np.array_equal(state[slot, :3 * channels].cpu().numpy().reshape(3, channels), rows.astype(np.float32))


def test_delta_prepare_of_more_tokens_than_a_launch_has_rows_of_tiles():
    """524,281 tokens of one span: one more than 65,535 tiles of eight hold."""
    from celeg_b200 import kernels
    tokens, dim, vw = 8 * 65535 + 1, 32, 4
    channels, stride = 2 * dim + vw, 2 * dim + vw + 4
    g = torch.Generator(device="cuda").manual_seed(8)
    proj, kernel = torch.randn(tokens, stride, device="cuda", generator=g), torch.randn(channels, 4, device="cuda", generator=g)
    state = torch.randn(1, 3 * channels, device="cuda", generator=g)
    rows = torch.cat([state.view(3, channels), proj[:, :channels]]).double()
    conv, gates = torch.zeros(tokens, channels, device="cuda"), torch.zeros(tokens, 2, device="cuda")
    span, begins = torch.zeros(tokens, dtype=torch.int32, device="cuda"), dev(np.array([0, tokens], dtype=np.int32))
    kernels.delta_prepare(proj, kernel, state, state.stride(0), span, begins, span[:1], conv, proj[:, channels:], proj[:, channels + 1:],
                          torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda"), gates, tokens, 1, channels, 4, 1, dim, 1, 1e-6)
    sums = sum(rows[j:j + tokens] * kernel[:, j].double() for j in range(4))
    want = sums * torch.sigmoid(sums)
    units = want[:, :2 * dim].view(tokens, 2, dim)
    units /= torch.sqrt(units.square().sum(-1, keepdim=True) + 1e-6)
    assert float((conv - want).abs().max()) < 10 * 2.0 ** -24 * float(sums.abs().max())      # (as above)
    assert float((gates[:, 0] - torch.sigmoid(proj[:, channels].double())).abs().max()) < 2e-6
    assert torch.equal(state.view(3, channels), rows[-3:].float())


@pytest.mark.parametrize("lengths", LENGTHS[2:])
@pytest.mark.parametrize("taps,channels,act", [(4, 516, 2), (3, 64, -1), (2, 33, 2)])
def test_channel_conv_in_tiles(lengths, taps, channels, act):
    from celeg_b200 import kernels
    rng = np.random.default_rng(taps + channels)
    tokens, requests = sum(lengths), len(lengths)
    proj = rng.normal(size=(tokens, channels + 4)).astype(np.float32)
    kernel, bias = rng.normal(size=(channels, taps)).astype(np.float32), rng.normal(size=channels).astype(np.float32)
    slots = list(rng.permutation(requests))
    carried = rng.normal(size=(requests, taps - 1, channels)).astype(np.float32)
    elements = (taps - 1) * channels
    state = torch.zeros((requests, -(-elements // 4) * 4), device="cuda")
    state[:, :elements] = dev(carried.reshape(requests, -1))
    span, begins = spans_of(lengths)
    out = torch.zeros((tokens, channels), device="cuda")
    kernels.channel_conv(dev(proj), dev(kernel), dev(bias), state, state.stride(0), span, begins, dev(np.array(slots, dtype=np.int32)),
                         out, tokens, requests, act)
    sums, carry = convolved(proj[:, :channels], kernel, carried, lengths, slots)
    want = silu(sums + bias) if act == 2 else sums + bias
    assert np.abs(out.cpu().numpy() - want).max() < 10 * 2.0 ** -24 * np.abs(sums).max()
    for slot, rows in carry.items():
        assert np.array_equal(state[slot, :elements].cpu().numpy().reshape(taps - 1, channels), rows.astype(np.float32))
