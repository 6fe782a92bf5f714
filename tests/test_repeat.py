"""Which layers may be repeated (no GPU)."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from inference_bench_b200.parts import base
from inference_bench_b200.parts.repeat import Repeat

T = torch.zeros(1, 4, 8)


@pytest.mark.parametrize("before,after,alike", [
    (None, None, True), (T, T.clone(), True), (None, T, False), (T, None, False), (T, torch.zeros(2, 4, 8), False),
    (base.NormedDelta(T, None), T, False), (base.NormedDelta(T, None), None, False), (T, base.NormedDelta(T, None), False), (base.ScaledDelta(T, 0.5), T, False),
    (base.SummedDelta(T, T), T, False), (base.NormedDelta(T, None), base.NormedDelta(T, None), False)])
def test_a_layer_is_repeated_behind_one_that_left_the_same_kind(before, after, alike):
    """Contributions of other arrangements among them: such a layer runs, and is not repeated."""
    block = SimpleNamespace(repeat_weights=lambda: [1, 2])
    cache = SimpleNamespace(c_view=lambda: None, tma=lambda: (None, 0))
    assert Repeat("key", block, cache, before).close(after) is alike
