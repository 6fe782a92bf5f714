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


def test_two_threads_note_their_own_layers(monkeypatch):
    """On one runtime, one thread's layer ends while another's is being noted: each keeps its own calls and buffers until its layers are repeated."""
    import threading

    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import lib
    from inference_bench_b200.parts.decoder import Decoder
    rt = SimpleNamespace(act_dtype=torch.float32, device="cpu")
    rt.empty = lambda shape: Runtime.empty(rt, shape)
    monkeypatch.setitem(lib._entry, "first", (lambda n: 0, 0))
    monkeypatch.setitem(lib._entry, "second", (lambda n: 0, 0))
    inside, other_done, reps = threading.Event(), threading.Event(), {}

    def layer(name, between):
        def forward(ctx, x, pending, cache):
            first = rt.empty((n,))
            lib.call(name, n)
            between()
            made[name] = [first, rt.empty((n,))]
            lib.call(name, n + 1)
            return T
        n = len(name)
        block = SimpleNamespace(repeat_weights=lambda: [1, 2], forward=forward, mixer=SimpleNamespace(position=SimpleNamespace(tables=lambda ctx: None)))
        cache = SimpleNamespace(c_view=lambda: None, tma=lambda: (None, 0))
        reps[name] = Decoder._noted(SimpleNamespace(rt=rt), block, None, T, cache, "key")[1]

    made = {}

    def other():
        inside.wait(10)
        layer("second", lambda: None)
        other_done.set()

    t = threading.Thread(target=other)
    t.start()
    layer("first", lambda: (inside.set(), other_done.wait(10)))
    t.join()
    for name in ("first", "second"):
        assert reps[name].calls == [(name, (len(name),)), (name, (len(name) + 1,))]
        assert [id(b) for b in reps[name].held] == [id(b) for b in made[name]]
