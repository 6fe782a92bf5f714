"""Layers that repeat the calls of the one before against the same layers run one by one (a traced step does that): the same bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _runner(dtype, head_dim, windows, page, qk_norm=True):
    from inference_bench_b200.cache.manager import CacheManager
    from inference_bench_b200.engine.model import plan_from_config
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.engine.step import ModelRunner
    from inference_bench_b200.parts.decoder import Decoder
    from inference_bench_b200.weights.random_init import random_weights
    cfg = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=333, hidden_size=256, intermediate_size=640, num_hidden_layers=len(windows), num_attention_heads=4,
               num_key_value_heads=2, head_dim=head_dim, rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=True, max_position_embeddings=4096, hidden_act="silu",
               attention_bias=False, torch_dtype="bfloat16")
    if any(windows):
        cfg.update(use_sliding_window=True, sliding_window=50, max_window_layers=0, layer_types=["sliding_attention" if w else "full_attention" for w in windows])
    rt = Runtime(DEV, dtype)
    decoder = Decoder(plan_from_config(cfg)[1])
    decoder.bind({k: v.to(DEV) for k, v in random_weights(decoder.weight_specs(), 4, std=0.06).items()}, rt)
    cache = CacheManager(decoder.cache_needs(), page, 200, 8, 1024, device=rt.device, dtype=rt.act_dtype, sources=decoder.cache_sources())
    return ModelRunner(decoder, cache, rt)


@pytest.mark.parametrize("dtype,head_dim,page", [("bfloat16", 128, 16), ("bfloat16", 64, 64), ("float32", 64, 16), ("bfloat16", 24, 8)])
@pytest.mark.parametrize("windows", [(0, 0, 0, 0, 0), (0, 1, 1, 1, 0, 0), (1, 0, 1, 0)])
def test_the_same_bits(dtype, head_dim, page, windows):
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.kernels import lib
    outs, counts = [], []
    for trace in (None, []):
        r = _runner(dtype, head_dim, windows, page)
        g = torch.Generator().manual_seed(9)
        got = []
        for i in range(4):
            r.cache.admit(i)
        # portions alone, decoded tokens beside them, many tokens (products that add to the stream themselves), decoded tokens alone
        for lens in ([5, 70, 0, 1], [1, 1, 33, 1], [300, 2, 200, 129], [1, 1, 1, 1], [0, 0, 3, 0]):
            entries = [StepEntry(i, torch.randint(0, 333, (n,), generator=g).tolist(), [0, n - 1]) for i, n in enumerate(lens) if n]
            before = lib.launches
            got.append(r.step(entries, trace=trace).clone())
            counts.append(lib.launches - before)
        outs.append((got, [gr.tensor.clone() for gr in r.cache.groups]))
    assert all(torch.equal(a, b) for a, b in zip(outs[0][0], outs[1][0]))
    assert all(torch.equal(a, b) for a, b in zip(outs[0][1], outs[1][1]))
    assert counts[:5] == counts[5:]


def test_a_shared_weight_is_not_repeated():
    """Two of a layer's weights at one address cannot be told apart: such layers run one by one."""
    from inference_bench_b200.engine.step import StepEntry
    outs = []
    for trace in (None, []):
        r = _runner("bfloat16", 128, (0, 0, 0, 0), 16)
        for b in r.decoder.blocks[:3]:
            b.mixer.k_norm = b.mixer.q_norm
        r.cache.admit(0)
        outs.append(r.step([StepEntry(0, list(range(40)), [39])], trace=trace).clone())
    assert torch.equal(*outs)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_layers_behind_one_of_another_arrangement(dtype):
    """A layer that gets a contribution with a norm of its own is not repeated; those behind it are."""
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.parts.standard import RMSNorm, SandwichBlock
    outs = []
    for trace in (None, []):
        r = _runner(dtype, 64, (0, 0, 0, 0, 0), 16)
        b, posts = r.decoder.blocks[0], [RMSNorm(f"post{i}", 256, 1e-6) for i in range(2)]
        for i, n in enumerate(posts):
            n.w = r.rt.vector(1 + 0.1 * torch.randn(256, generator=torch.Generator().manual_seed(i)))
        r.decoder.blocks[0] = SandwichBlock(b.mixer_norm, b.mixer, b.feed_forward_norm, b.feed_forward, *posts)
        r.cache.admit(0)
        outs.append([r.step([StepEntry(0, list(range(n)), [n - 1])], trace=trace).clone() for n in (40, 1, 300)])
    assert all(torch.equal(a, b) for a, b in zip(*outs))
