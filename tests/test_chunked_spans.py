"""The bound on the chunks of a step: a step with more short spans than the scratch has room for is told so beforehand."""

from types import SimpleNamespace

import pytest
import torch


@pytest.mark.parametrize("tokens,spans,single", ((0, 0, 0), (2048, 1, 0), (2048, 87, 0), (2048, 88, 0), (2050, 90, 2), (2051, 91, 2)))
def test_fits_agrees_with_of(monkeypatch, tokens, spans, single):
    from celeg_b200 import kernels
    from celeg_b200.parts.decayed import ChunkedSpans
    monkeypatch.setattr(kernels, "chunk_tokens", lambda: 64)
    monkeypatch.setattr(kernels, "chunk_plan", lambda *args: None)
    rt = SimpleNamespace(max_tokens=2048, max_requests=8,
                         flat_scratch=lambda name, elements, dtype: torch.zeros(elements, dtype=dtype))
    held = ChunkedSpans(rt)
    step = SimpleNamespace(tokens=tokens, spans=spans, span_begin=torch.zeros(spans + 1, dtype=torch.int32), extras={})
    fits = held.fits(step, single)
    assert fits == ((tokens - single) // 64 + spans - single <= 32 + 8 + 48)
    if fits:
        assert held.of(step, single)[1:] == (spans - single, (tokens - single) // 64 + spans - single)
    else:
        with pytest.raises(ValueError):
            held.of(step, single)
