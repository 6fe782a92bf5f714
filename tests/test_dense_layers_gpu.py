"""Layers launched by one call each (csrc/dense_layer.cu) against the same layers run by their parts: the same bits, over the forms their products take."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _runner(hidden, inter, heads, kv_heads, head_dim, window, page, options=None, layers=3, change=lambda plan: plan):
    from inference_bench_b200.cache.manager import CacheManager
    from inference_bench_b200.config.runtime_options import RuntimeOptions
    from inference_bench_b200.engine.model import plan_from_config
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.engine.step import ModelRunner
    from inference_bench_b200.parts.decoder import Decoder
    from inference_bench_b200.weights.random_init import random_weights
    cfg = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=333, hidden_size=hidden, intermediate_size=inter, num_hidden_layers=layers, num_attention_heads=heads,
               num_key_value_heads=kv_heads, head_dim=head_dim, rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=True, max_position_embeddings=8192, hidden_act="silu",
               attention_bias=False, torch_dtype="bfloat16")
    if window:
        cfg.update(use_sliding_window=True, sliding_window=window, max_window_layers=0, layer_types=["full_attention", "sliding_attention"] * (layers // 2) + ["full_attention"] * (layers % 2))
    rt = Runtime(DEV, "bfloat16", options=options or RuntimeOptions())
    decoder = Decoder(change(plan_from_config(cfg)[1]))
    decoder.bind({k: v.to(DEV) for k, v in random_weights(decoder.weight_specs(), 5, std=0.05).items()}, rt)
    cache = CacheManager(decoder.cache_needs(), page, 12000 // page, 8, 6000, device=rt.device, dtype=rt.act_dtype, sources=decoder.cache_sources())
    return ModelRunner(decoder, cache, rt)


# tokens of up to three requests a step: around the token tiles of the products (16, 32, 64, 128), where the q/k/v product takes its epilogue and the
# cost model changes forms, the largest step that goes this way and one beyond it; single tokens beside portions in most of them
STEPS = [[2], [15, 1, 1], [17, 16], [31, 1, 33], [63, 1, 1], [65], [127, 1, 1], [129], [300, 1, 7], [1000, 1, 1], [1, 1, 1], [2558, 1, 1], [1, 2560]]


@pytest.mark.parametrize("sizes", [(256, 640, 4, 2, 64, 0, 16), (256, 640, 2, 2, 128, 70, 8), (1024, 3072, 16, 8, 128, 0, 64), (320, 9728, 4, 1, 128, 0, 128)])
def test_the_same_bits_as_the_parts(sizes, monkeypatch):
    """Three ways: one call a layer, the same launches one by one for somebody who looks at them, and the parts."""
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.kernels import dense, lib
    from inference_bench_b200.parts.standard import PreNormBlock
    outs, counts, native, by_parts = [], [], [], []
    forward = PreNormBlock.forward
    monkeypatch.setattr(PreNormBlock, "forward", lambda self, ctx, *a: (by_parts.append(ctx.n_tokens), forward(self, ctx, *a))[1])
    for way in ("native", "watched", "parts"):
        names = []
        if way == "native":
            counted = lib.call_counted
            monkeypatch.setattr(lib, "call_counted", lambda name, *a: (native.append(name), counted(name, *a))[1])
        elif way == "watched":
            real = lib.call
            monkeypatch.setattr(lib, "call", lambda name, *a: (names.append(name), real(name, *a))[1])
        else:
            monkeypatch.setattr(dense, "MAX_TOKENS", 0)
        r, g = _runner(*sizes), torch.Generator().manual_seed(3)
        for i in range(3):
            r.cache.admit(i)
        got = []
        del by_parts[:]
        for lens in STEPS:
            entries = [StepEntry(i, torch.randint(0, 333, (n,), generator=g).tolist(), [0, n - 1]) for i, n in enumerate(lens)]
            before = lib.launches
            got.append(r.step(entries).clone())
            counts.append(lib.launches - before)
        outs.append(got + [gr.tensor.clone() for gr in r.cache.groups])
        assert way != "watched" or "ib_attention_prefill_ws" in names
        assert way == "parts" or set(by_parts) == {3, 2561}   # every step but the one of single tokens and the one of 2,561
    assert native.count("ib_dense_layer") == 3 * 11
    assert counts[:len(STEPS)] == counts[len(STEPS):2 * len(STEPS)] == counts[2 * len(STEPS):]
    assert all(torch.equal(a, b) and torch.equal(a, c) for a, b, c in zip(*outs))


@pytest.mark.parametrize("options", [dict(prefill_attention="tcgen05"), dict(decode_attention="split"), dict(gemm="simt")])
def test_other_kernels_asked_for_run(options, monkeypatch):
    """A runtime that asks for kernels this way does not have keeps its parts."""
    from inference_bench_b200.config.runtime_options import RuntimeOptions
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.kernels import lib
    monkeypatch.setattr(lib, "call_counted", lambda *a: pytest.fail("a layer went past its parts"))
    r = _runner(256, 640, 4, 2, 64, 0, 16, RuntimeOptions(**options))
    r.cache.admit(0)
    assert torch.isfinite(r.step([StepEntry(0, list(range(40)), [39])])).all()


def test_a_refused_kernel_ends_the_layer(monkeypatch):
    """Nothing is launched behind a product that was refused: the request's pages and the count of kernels stay as they were before it."""
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.kernels import gemm_tcgen05 as G, lib
    r = _runner(256, 640, 4, 2, 64, 0, 16)
    r.cache.admit(0)
    r.step([StepEntry(0, list(range(40)), [39])])
    before = [g.tensor.clone() for g in r.cache.groups]
    form = G.product_form
    monkeypatch.setattr(G, "product_form", lambda rt, T, n, k, allow_split=True, add=False: form(rt, T, n, k, allow_split, add) if add else ("single", 17, 1, False))
    with pytest.raises(lib.KernelError, match="token tile 17"):
        r.step([StepEntry(0, list(range(50)), [49])])
    monkeypatch.undo()
    torch.cuda.synchronize()
    assert all(torch.equal(a, g.tensor) for a, g in zip(before, r.cache.groups))
    assert r.cache.length(0) == 40
    assert torch.isfinite(r.step([StepEntry(0, list(range(50)), [49])])).all()


def test_layers_of_two_keys_around_other_arrangements(monkeypatch):
    """Full and windowed layers before, between and behind layers with another norm (which the parts run): the same bits as by parts alone."""
    from dataclasses import replace
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.kernels import dense, lib

    def other(plan):   # layers 1 and 4 of six
        norm = lambda spec: replace(spec, kind="layernorm")
        return replace(plan, layers=tuple(replace(lp, mixer_norm=norm(lp.mixer_norm), feed_forward_norm=norm(lp.feed_forward_norm)) if i in (1, 4) else lp
                                          for i, lp in enumerate(plan.layers)))
    outs, native, counted = [], [], lib.call_counted
    monkeypatch.setattr(lib, "call_counted", lambda name, *a: (native.append(name), counted(name, *a))[1])
    for way in ("native", "parts"):
        if way == "parts":
            monkeypatch.setattr(dense, "MAX_TOKENS", 0)
        r, g = _runner(256, 640, 4, 2, 64, 70, 16, layers=6, change=other), torch.Generator().manual_seed(7)
        for i in range(2):
            r.cache.admit(i)
        got = [r.step([StepEntry(i, torch.randint(0, 333, (n,), generator=g).tolist(), [0, n - 1]) for i, n in enumerate(lens)]).clone() for lens in ([90, 33], [1, 40], [200, 1])]
        outs.append(got + [gr.tensor.clone() for gr in r.cache.groups])
    assert len(native) == 3 * 4
    assert all(torch.equal(a, b) for a, b in zip(*outs))
