"""Which steps go in chunks of 64 tokens (parts.recurrent.PortionsInChunks): the rule over portions of many lengths, the bounds
on the chunks that scratch and launches are sized by, and the launch shapes of padded steps, which hold for one answer only."""
from __future__ import annotations

import random
from types import SimpleNamespace

import pytest
import torch

from celeg_b200 import kernels
from celeg_b200.parts.recurrent import GatedDeltaMixer, GeneralDeltaMixer, MlstmMixer, PortionsInChunks, RetentionMixer

MIXERS = (MlstmMixer, RetentionMixer, GatedDeltaMixer, GeneralDeltaMixer)


@pytest.fixture(autouse=True)
def on_the_host(monkeypatch):
    monkeypatch.setattr(kernels, "chunk_tokens", lambda: 64)
    monkeypatch.setattr(kernels, "chunk_plan", lambda *args: None)


def rule_of(mixer, max_tokens=1 << 14, max_requests=8):
    rt = SimpleNamespace(max_tokens=max_tokens, max_requests=max_requests, portion_rules={},
                         flat_scratch=lambda name, elements, dtype: torch.zeros(elements, dtype=dtype))
    part = PortionsInChunks()
    part.CHUNKED_FROM, part.TOKENS_A_CHUNK = mixer.CHUNKED_FROM, mixer.TOKENS_A_CHUNK
    part.plan_chunks(rt)
    return part, rt


def step_of(lengths, single=0, known=True):
    lengths = [1] * single + list(lengths)
    return SimpleNamespace(tokens=sum(lengths), spans=len(lengths), leading_single_tokens=single, max_span=max(lengths), extras={},
                           span_begin=torch.zeros(len(lengths) + 1, dtype=torch.int32), host_span_lengths=lengths if known else None)


@pytest.mark.parametrize("mixer", MIXERS)
def test_many_short_portions_go_token_by_token(mixer):
    """As measured: eight, 16 and 48 portions of 4 and 20 tokens, and a portion just long enough among forty of eight."""
    rule, _ = rule_of(mixer)
    for count in (8, 16, 48):
        for each in (4, 20):
            assert not rule.in_chunks([each] * count) and rule.leading(step_of([each] * count, 2)) == 2 + each * count
    assert not rule.in_chunks([160] + [8] * 40) and not rule.in_chunks([]) and not rule.in_chunks([mixer.CHUNKED_FROM - 1])


@pytest.mark.parametrize("mixer", MIXERS)
def test_long_portions_go_in_chunks(mixer):
    rule, _ = rule_of(mixer)
    for lengths in ([mixer.CHUNKED_FROM], [2048], [500] * 16, [1500] + [30] * 16, [1, 2000, 3]):
        assert rule.in_chunks(lengths)
        for known in (True, False):        # (without the lengths, their longest and the most chunks they may make)
            assert rule.leading(step_of(lengths, 3, known)) == 3
    assert rule_of(MlstmMixer)[0].in_chunks([150] * 48) and rule_of(RetentionMixer)[0].in_chunks([600] + [20] * 40)
    assert not rule_of(GeneralDeltaMixer)[0].in_chunks([600] + [20] * 40)


@pytest.mark.parametrize("mixer", MIXERS)
def test_scratch_and_launches_hold_the_chunks_of_every_step_that_goes_in_chunks(mixer):
    rng, taken = random.Random(1), 0
    for _ in range(3000):
        max_tokens = rng.choice([mixer.CHUNKED_FROM, 500, 512, 2048, 8192])
        lengths, left = [], max_tokens - rng.randint(0, max_tokens // 2)
        while left > 0 and len(lengths) < 200:
            lengths.append(min(left, rng.choice([1, 2, rng.randint(1, 70), rng.randint(100, 1000), left])))
            left -= lengths[-1]
        rule, _ = rule_of(mixer, max_tokens)
        if rule.spans is None or not rule.in_chunks(lengths):
            continue
        taken += 1
        _, spans, chunks = rule.spans.of(step_of(lengths), 0)
        assert spans == len(lengths) and sum(-(-n // 64) for n in lengths) <= chunks <= rule.spans.chunks_held <= rule.spans.max_chunks
        assert rule.spans.plan.numel() >= rule.spans.max_chunks + spans + 2
    assert taken > 300


def test_scratch_does_not_grow_with_requests_and_is_none_where_no_step_is_long_enough():
    held = [rule_of(GeneralDeltaMixer, 2208, requests)[0].spans.chunks_held for requests in (8, 256)]
    assert held[0] == held[1] == 55
    rule, rt = rule_of(GeneralDeltaMixer, 64)
    assert rule.spans is None and not rt.portion_rules and rule.leading(step_of([40, 20], 2)) == 62


def test_padded_steps_share_a_launch_shape_only_where_the_answers_agree():
    from celeg_b200.engine.step import StepFunction
    rule, rt = rule_of(MlstmMixer)
    other, _ = rule_of(GeneralDeltaMixer)

    def key_of(lengths, rules):
        runtime = SimpleNamespace(portion_routes=lambda portions: tuple(r.in_chunks(portions) for r in rules))
        self = SimpleNamespace(use_graphs=True, max_spans=64, padded_single_rows=lambda n: 4, rt=runtime, page_tokens=16, max_pages=64,
                               storage=SimpleNamespace(scratch_page_count=32), buffer_tokens=4096, span_capacity=104, _graphs={},
                               _prompt_seen={}, max_padded_graphs=4)
        entries = [SimpleNamespace(tokens=[0] * n) for n in [1, 1, 1] + lengths]
        for _ in range(8):
            shape = StepFunction._padded_prompt_shape(self, entries, len(lengths), 600)
            if shape is not None:
                return shape.key
        raise AssertionError("the shape never came often enough")

    long, short, longest = [300, 10, 10, 10], [90, 80, 80, 80], [560, 10, 10, 10]
    assert key_of(long, []) == key_of(short, [])
    assert key_of(long, [rule]) != key_of(short, [rule]) and key_of(long, [other]) == key_of(short, [other])
    assert rule.in_chunks(longest) and key_of(longest, [rule, other]) != key_of([150, 150, 150, 140], [rule, other])
