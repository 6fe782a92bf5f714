"""The work that a user of the engine has it do, as cases that can be timed and checked one by one.

Two kinds go through whole steps of a few-layer model: "decode" (one captured step of single tokens, tokens in from the host and logits of
every row out) and "portion" (one step of prompt portions, alone or beside decoded tokens). Three kinds are one sublayer of another served
architecture with the norm in front of it and the norm that adds its output to the stream, on prompt portions: "latent" (latent attention),
"experts" (routed experts) and "recurrence" (a gated linear recurrence). Weights, tokens and rows are made from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda:0"
EPS = 1e-6

# Layer sizes of the Qwen3 shapes that the engine's benchmark runs; the vocabulary is the full one only where its share of a step is the point.
SHAPES = {
    "0.6b": dict(hidden=1024, inter=3072, heads=16, kv_heads=8, tied=True),
    "8b": dict(hidden=4096, inter=12288, heads=32, kv_heads=8, tied=False),
}
HEAD_DIM = 128
# Sublayer sizes of the benchmark's other designs.
LATENT = {
    "small": dict(width=1024, heads=8, dim=64, rot=32, vdim=64, rank=256),
    "lite": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, rank=512),
}
EXPERTS = {
    "small": dict(width=1024, experts=16, top=2, ff=1024, shared=1024, groups=2, keep=1),
    "lite": dict(width=2048, experts=64, top=6, ff=1408, shared=2816, groups=8, keep=4),
}
RECURRENCE = {
    "small": dict(width=1024, heads=8, dim=128, vdim=128),
    "mid": dict(width=2048, heads=16, dim=128, vdim=128),
}


def listed():
    return [
        # one user's chat on the smallest shape: a step is many small launches, and latency is all that counts
        dict(name="decode_b1_small", kind="decode", shape="0.6b", layers=12, vocab=151936, batch=1, context=600, page=64),
        # the engine's headline workload: eight requests around 2,048 tokens, page size 16
        dict(name="decode_b8", kind="decode", shape="8b", layers=5, vocab=32768, batch=8, context=2200, page=16),
        # a full server: 64 requests at contexts from short to long, half of the step's bytes are keys and values
        dict(name="decode_b64", kind="decode", shape="8b", layers=3, vocab=32768, batch=64, context=3000, page=64),
        # a long prompt's portion of the default size
        dict(name="prefill_2048", kind="portion", shape="8b", layers=3, vocab=32768, prompts=1, tokens=2048, past=0, rows=0, dtype="bfloat16"),
        # three prompts of odd lengths that arrive together
        dict(name="prefill_ragged", kind="portion", shape="8b", layers=2, vocab=32768, prompts=3, tokens=1003, past=0, rows=0, dtype="bfloat16"),
        # a follow-up question of a chat: a short portion behind a cached context
        dict(name="prefill_followup", kind="portion", shape="0.6b", layers=8, vocab=32768, prompts=1, tokens=61, past=900, rows=0, dtype="bfloat16"),
        # the mixed step of a busy server: eight portions of 512 tokens, some far into their prompts, beside 56 decoded tokens
        dict(name="mixed_step", kind="portion", shape="8b", layers=2, vocab=32768, prompts=8, tokens=4096, past=1200, rows=56, dtype="bfloat16"),
        # the true 32-bit path, on which logits are checked against other implementations
        dict(name="float32_prompt", kind="portion", shape="0.6b", layers=4, vocab=32768, prompts=2, tokens=777, past=0, rows=0, dtype="float32"),
        # latent attention over a long prompt's portion
        dict(name="latent_2048", kind="latent", size="lite", prompts=1, tokens=2048, past=0),
        # latent attention over short portions of several requests behind cached contexts
        dict(name="latent_ragged", kind="latent", size="lite", prompts=3, tokens=333, past=700),
        # routed experts with a shared one over a long prompt's portion
        dict(name="experts_2048", kind="experts", size="lite", prompts=1, tokens=2048),
        # the recurrence over a long prompt's portion, behind an earlier one
        dict(name="recurrence_2048", kind="recurrence", size="mid", prompts=1, tokens=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "portion", "portion", "portion", "float32", "latent", "experts", "recurrence"])
    if kind == "decode":
        shape = rng.choice(["0.6b", "8b"])
        return dict(kind="decode", shape=shape, layers=8 if shape == "0.6b" else 3, vocab=32768, batch=_log_int(rng, 1, 64), context=_log_int(rng, 64, 3000),
                    page=rng.choice([16, 64]))
    if kind == "portion":
        prompts = rng.choice([1, 1, 2, 3, 5])
        return dict(kind="portion", shape=rng.choice(["0.6b", "8b"]), layers=2, vocab=32768, prompts=prompts, tokens=max(2 * prompts, _log_int(rng, 12, 4096)),
                    past=rng.choice([0, _log_int(rng, 16, 1200)]), rows=rng.choice([0, 0, _log_int(rng, 1, 56)]), dtype="bfloat16")
    if kind == "float32":
        return dict(kind="portion", shape="0.6b", layers=rng.choice([1, 2, 3]), vocab=32768, prompts=rng.choice([1, 2]), tokens=_log_int(rng, 8, 900), past=0, rows=0,
                    dtype="float32")
    prompts = rng.choice([1, 1, 2, 4])
    tokens = max(2 * prompts, _log_int(rng, 24, 2048))
    if kind == "latent":
        return dict(kind="latent", size=rng.choice(["small", "lite"]), prompts=prompts, tokens=tokens, past=rng.choice([0, _log_int(rng, 16, 900)]))
    if kind == "experts":
        return dict(kind="experts", size=rng.choice(["small", "lite"]), prompts=prompts, tokens=tokens)
    return dict(kind="recurrence", size=rng.choice(["small", "mid"]), prompts=prompts, tokens=tokens)


# ---------------------------------------------------------------------------------------------- sizes and inputs of a case
def _split(total, parts):
    """`total` tokens over `parts` requests, unevenly: 1 : 2 : 3 ... (every request gets one at least)."""
    weights = np.arange(1, parts + 1)
    cuts = np.maximum(1, np.floor(total * weights / weights.sum())).astype(int)
    cuts[-1] += total - int(cuts.sum())
    return cuts.tolist()


def _portions(case):
    """(tokens, cached tokens before them) of every request of a step: the prompt portions, then the decoded tokens."""
    n, past = case["prompts"], case.get("past", 0)
    if case.get("rows", 0):   # beside decoded tokens the scheduler cuts equal portions
        sizes = [case["tokens"] // n + (1 if i < case["tokens"] % n else 0) for i in range(n)]
    else:
        sizes = _split(case["tokens"], n)
    out = [(t, past * (2 * i + 1) // (2 * n) if n > 1 else past) for i, t in enumerate(sizes)]
    return out + [(1, c) for c in _contexts(case.get("rows", 0), 2000)]


def _contexts(batch, longest):
    """Contexts of `batch` requests, spread evenly between a quarter of the longest and the longest; eight or fewer lie close together."""
    if batch <= 8:
        return [longest - (longest // 16) * i // max(1, batch) - i for i in range(batch)]
    return [longest // 4 + (longest - longest // 4) * ((i * 37) % batch) // batch for i in range(batch)]


def _generator(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _normal(shape, std, seed, salt, dtype=torch.float32):
    return (torch.randn(shape, generator=_generator(seed, salt), device=DEV, dtype=torch.float32) * std).to(dtype)


def _make(specs, seed):
    """{name: tensor} for [(name, shape, std or (mean, std))]: matrices in bfloat16, vectors in float32."""
    out = {}
    for i, (name, shape, how) in enumerate(specs):
        if isinstance(how, tuple):
            out[name] = how[0] + _normal(shape, how[1], seed, 17 + i)
        else:
            out[name] = _normal(shape, how, seed, 17 + i, torch.bfloat16)
    return out


def _token_ids(seed, n, vocab):
    return np.random.default_rng(seed).integers(0, vocab, size=n).tolist()


def _sequences(case, seed):
    """Every request's whole token sequence: what is cached before the step, then the step's tokens."""
    if case["kind"] == "decode":
        lens = [c + 1 for c in _contexts(case["batch"], case["context"])]
    else:
        lens = [t + p for t, p in _portions(case)]
    return [_token_ids(seed * 1009 + i, n, case["vocab"]) for i, n in enumerate(lens)]


# ---------------------------------------------------------------------------------------------- whole steps of a few-layer model
def _qwen3_config(case):
    s = SHAPES[case["shape"]]
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=case["vocab"], hidden_size=s["hidden"], intermediate_size=s["inter"],
                num_hidden_layers=case["layers"], num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"], head_dim=HEAD_DIM, rms_norm_eps=EPS,
                rope_theta=1000000.0, tie_word_embeddings=s["tied"], max_position_embeddings=40960, hidden_act="silu", attention_bias=False, torch_dtype="bfloat16")


def _qwen3_specs(case):
    s = SHAPES[case["shape"]]
    H, I, q, kv = s["hidden"], s["inter"], s["heads"] * HEAD_DIM, s["kv_heads"] * HEAD_DIM
    specs = [("model.embed_tokens.weight", (case["vocab"], H), 0.02), ("model.norm.weight", (H,), (1.0, 0.1))]
    if not s["tied"]:
        specs.append(("lm_head.weight", (case["vocab"], H), 0.02))
    for i in range(case["layers"]):
        p = f"model.layers.{i}"
        specs += [(f"{p}.input_layernorm.weight", (H,), (1.0, 0.1)), (f"{p}.post_attention_layernorm.weight", (H,), (1.0, 0.1)),
                  (f"{p}.self_attn.q_norm.weight", (HEAD_DIM,), (1.0, 0.1)), (f"{p}.self_attn.k_norm.weight", (HEAD_DIM,), (1.0, 0.1)),
                  (f"{p}.self_attn.q_proj.weight", (q, H), 0.02), (f"{p}.self_attn.k_proj.weight", (kv, H), 0.02), (f"{p}.self_attn.v_proj.weight", (kv, H), 0.02),
                  (f"{p}.self_attn.o_proj.weight", (H, q), 0.02), (f"{p}.mlp.gate_proj.weight", (I, H), 0.02), (f"{p}.mlp.up_proj.weight", (I, H), 0.02),
                  (f"{p}.mlp.down_proj.weight", (H, I), 0.02)]
    return specs


def _prepare_model(case, seed):
    """A bound model with its cache, and the requests' contexts run into it in portions."""
    from inference_bench_b200.cache.manager import CacheManager
    from inference_bench_b200.engine.executor import GpuExecutor
    from inference_bench_b200.engine.model import plan_from_config
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.engine.step import ModelRunner, StepEntry
    from inference_bench_b200.parts.decoder import Decoder
    from inference_bench_b200.sampling.params import GREEDY
    seqs = _sequences(case, seed)
    news = [1] * len(seqs) if case["kind"] == "decode" else [t for t, _ in _portions(case)]
    page = case.get("page", 64)
    rt = Runtime(DEV, case.get("dtype", "bfloat16"))
    _, plan = plan_from_config(_qwen3_config(case))
    decoder = Decoder(plan)
    decoder.bind(_make(_qwen3_specs(case), seed), rt)
    longest = max(len(s) for s in seqs)
    pages = sum(-(-len(s) // page) for s in seqs)
    cache = CacheManager(decoder.cache_needs(), page, pages, len(seqs), longest, device=rt.device, dtype=rt.act_dtype, sources=decoder.cache_sources())
    runner = ModelRunner(decoder, cache, rt)
    batch, held = [], 0
    for rid, (seq, new) in enumerate(zip(seqs, news)):   # contexts in steps of up to about 8,192 tokens
        cache.admit(rid)
        if len(seq) > new:
            batch.append(StepEntry(rid, seq[:len(seq) - new], []))
            held += len(seq) - new
        if held >= 8192 or (batch and rid == len(seqs) - 1):
            runner.step(batch, check=False)
            batch, held = [], 0
    entries = [StepEntry(rid, seq[len(seq) - new:], [new - 1]) for rid, (seq, new) in enumerate(zip(seqs, news))]
    state = dict(kind=case["kind"], runner=runner, cache=cache, entries=entries, sampling=[(GREEDY, 0)] * len(entries))
    if case["kind"] == "decode":
        state["executor"] = GpuExecutor(runner)
        state["executor"].graph_for(len(entries))
    return state


def _run_model(state):
    cache, entries = state["cache"], state["entries"]
    if state["kind"] == "decode":
        state["executor"].execute(entries, state["sampling"])
        logits = state["executor"].last_logits[:len(entries)]
    else:
        logits = state["runner"].step(entries, check=False)
    for e in entries:   # the same step again: the requests go back to where they were
        cache.commit(e.request, cache.length(e.request) - len(e.tokens))
    return {"logits": logits, "cache": [g.tensor for g in cache.groups]}


def _rms(x, w, eps=EPS):
    return w * (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps))


def _turn_half(x, pos, theta):
    """x [T, heads, D]: entry i turned with entry i + D/2."""
    D = x.shape[-1]
    inv = 1.0 / theta ** (torch.arange(0, D, 2, dtype=torch.float64, device=DEV) / D)
    a = pos.to(torch.float64)[:, None, None] * inv
    c, s, lo, hi = torch.cos(a), torch.sin(a), x[..., :D // 2], x[..., D // 2:]
    return torch.cat([lo * c - hi * s, hi * c + lo * s], dim=-1)


def _attend(q, k, v, first, scale):
    """q [T, heads, D] at positions first .. first + T - 1 against k, v [keys, kv_heads, D]."""
    T, heads, _ = q.shape
    group = heads // k.shape[1]
    out = torch.empty((T, heads, v.shape[-1]), dtype=q.dtype, device=q.device)
    hidden = torch.arange(k.shape[0], device=DEV)[None, :] > (first + torch.arange(T, device=DEV))[:, None]
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T) * scale
        out[:, h] = torch.softmax(s.masked_fill(hidden, -math.inf), dim=-1) @ v[:, h // group]
    return out


def _exact_model(case, seed):
    s, W = SHAPES[case["shape"]], {k: v.double() for k, v in _make(_qwen3_specs(case), seed).items()}
    heads, kvh, head = s["heads"], s["kv_heads"], W["model.embed_tokens.weight" if s["tied"] else "lm_head.weight"]
    rows = []
    for seq in _sequences(case, seed):
        n = len(seq)
        x = W["model.embed_tokens.weight"][torch.tensor(seq, device=DEV)]
        pos = torch.arange(n, device=DEV)
        for i in range(case["layers"]):
            p, first = f"model.layers.{i}", n - 1 if i == case["layers"] - 1 else 0   # the last layer is needed at the last position only
            a = f"{p}.self_attn"
            h = _rms(x, W[f"{p}.input_layernorm.weight"])
            k = _turn_half(_rms((h @ W[f"{a}.k_proj.weight"].T).view(n, kvh, HEAD_DIM), W[f"{a}.k_norm.weight"]), pos, 1e6)
            v = (h @ W[f"{a}.v_proj.weight"].T).view(n, kvh, HEAD_DIM)
            q = _turn_half(_rms((h[first:] @ W[f"{a}.q_proj.weight"].T).view(n - first, heads, HEAD_DIM), W[f"{a}.q_norm.weight"]), pos[first:], 1e6)
            o = _attend(q, k, v, first, HEAD_DIM ** -0.5).reshape(n - first, heads * HEAD_DIM)
            x = x[first:] + o @ W[f"{a}.o_proj.weight"].T
            h = _rms(x, W[f"{p}.post_attention_layernorm.weight"])
            x = x + (torch.nn.functional.silu(h @ W[f"{p}.mlp.gate_proj.weight"].T) * (h @ W[f"{p}.mlp.up_proj.weight"].T)) @ W[f"{p}.mlp.down_proj.weight"].T
        rows.append(_rms(x[-1], W["model.norm.weight"]) @ head.T)
    return {"logits": torch.stack(rows), "cache": [None]}


def _work_model(case):
    s = SHAPES[case["shape"]]
    H, I, q, kv = s["hidden"], s["inter"], s["heads"] * HEAD_DIM, s["kv_heads"] * HEAD_DIM
    layer = (q + 2 * kv) * H + H * q + 3 * I * H
    steps = [(1, c) for c in _contexts(case["batch"], case["context"])] if case["kind"] == "decode" else _portions(case)
    size = 4 if case.get("dtype") == "float32" else 2
    T, n = sum(t for t, _ in steps), len(steps)
    pairs = sum(t * p + t * (t + 1) / 2 for t, p in steps)
    flops = 2.0 * T * case["layers"] * layer + case["layers"] * 4.0 * pairs * q + 2.0 * n * case["vocab"] * H
    nbytes = size * (case["layers"] * layer + case["vocab"] * H + T * H) + size * case["layers"] * 2 * kv * sum(t + p for t, p in steps) + 4.0 * n * case["vocab"]
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------- one sublayer on prompt portions
def _sublayer_specs(case):
    if case["kind"] == "latent":
        z = LATENT[case["size"]]
        W, H, D, R, V, r = z["width"], z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
        own = [("m.q", (H * (D + R), W), W ** -0.5), ("m.dkv", (r + R, W), W ** -0.5), ("m.dkv.norm", (r,), (1.0, 0.1)), ("m.uk", (H * D, r), r ** -0.5),
               ("m.uv", (H * V, r), r ** -0.5), ("m.o", (W, H * V), (H * V) ** -0.5)]
    elif case["kind"] == "experts":
        z = EXPERTS[case["size"]]
        W, F, S = z["width"], z["ff"], z["shared"]
        own = [("m.router", (z["experts"], W), W ** -0.5)]
        for k in range(z["experts"]):
            own += [(f"m.e{k}.gate", (F, W), W ** -0.5), (f"m.e{k}.up", (F, W), W ** -0.5), (f"m.e{k}.down", (W, F), 4 * F ** -0.5)]
        own += [("m.shared.gate", (S, W), W ** -0.5), ("m.shared.up", (S, W), W ** -0.5), ("m.shared.down", (W, S), S ** -0.5)]
    else:
        z = RECURRENCE[case["size"]]
        W, H, D, V = z["width"], z["heads"], z["dim"], z["vdim"]
        own = [("m.q", (H * D, W), W ** -0.5), ("m.f", (H * D, W), W ** -0.5), ("m.f.b", (H * D,), (1.0, 0.5)), ("m.lower", (H * D,), (0.5, 0.1)),
               ("m.v", (H * V, W), W ** -0.5), ("m.norm", (V,), (1.0, 0.1)), ("m.o", (W, H * V), (H * V) ** -0.5)]
    return z, [("n1", (W,), (1.0, 0.1)), ("n2", (W,), (1.0, 0.1))] + own


def _prepare_sublayer(case, seed):
    from inference_bench_b200.cache.manager import CacheManager
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.parts.experts import RoutedExperts
    from inference_bench_b200.parts.latent import LatentAttention
    from inference_bench_b200.parts.recurrent import GatedLinearRecurrence
    from inference_bench_b200.parts.standard import RMSNorm, RotaryEmbedding
    z, specs = _sublayer_specs(case)
    W = z["width"]
    rt = Runtime(DEV, "bfloat16")
    if case["kind"] == "latent":
        part = LatentAttention("m", W, z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"], (z["dim"] + z["rot"]) ** -0.5, EPS,
                               RotaryEmbedding(z["rot"], 1e4, pairing="interleaved"))
    elif case["kind"] == "experts":
        part = RoutedExperts("m", W, z["ff"], z["experts"], z["top"], groups=z["groups"], groups_keep=z["keep"], shared_ff=z["shared"])
    else:
        part = GatedLinearRecurrence("m", W, z["heads"], z["dim"], z["vdim"], EPS)
    norm_in, norm_out = RMSNorm("n1", W, EPS), RMSNorm("n2", W, EPS)
    weights = _make(specs, seed)
    for p in (part, norm_in, norm_out):
        p.bind(weights, rt)
    cache = None
    sizes = _portions(case)
    if case["kind"] != "experts":
        longest = max(t + p for t, p in sizes)
        cache = CacheManager([part.cache_need()], 64, sum(-(-(t + p) // 64) for t, p in sizes), len(sizes), longest, device=rt.device, dtype=rt.act_dtype)
        for rid, (t, p) in enumerate(sizes):
            cache.admit(rid)
            cache.extend(rid, p)
            cache.commit(rid, p)
    state = dict(kind=case["kind"], rt=rt, part=part, norm_in=norm_in, norm_out=norm_out, cache=cache, sizes=sizes, x=_normal((case["tokens"], W), 1.0, seed, 5))
    if case["kind"] == "recurrence":   # what earlier portions left
        cache.states[0].tensor.copy_(_past_state(case, seed))
    if case["kind"] == "latent" and case["past"]:
        for rid, (rows, (t, p)) in enumerate(zip(_past_rows(case, seed), sizes)):
            pool, table = cache.groups[0].tensor, cache.table(0, rid)
            for at in range(0, p, 64):
                n = min(64, p - at)
                pool[0, int(table[at // 64]), 0, 0, :n] = rows[at:at + n]
    return state


def _past_state(case, seed):
    z = RECURRENCE[case["size"]]
    return _normal((case["prompts"] + 1, z["heads"], z["dim"], z["vdim"]), 0.5, seed, 7)


def _past_rows(case, seed):
    """The cached rows before every request's portion: bfloat16, around one like the normed latents."""
    z = LATENT[case["size"]]
    return [_normal((p, z["rank"] + z["rot"]), 1.0, seed, 1000 + i, torch.bfloat16) for i, (_, p) in enumerate(_portions(case))]


def _run_sublayer(state):
    from inference_bench_b200.engine.context import Segment, build_context
    rt, part, cache, sizes = state["rt"], state["part"], state["cache"], state["sizes"]
    x = state["x"].clone()
    if cache is None:
        views = None
        segments = [Segment(i, i, p, [0] * t) for i, (t, p) in enumerate(sizes)]
    else:
        for i, (t, p) in enumerate(sizes):
            cache.extend(i, p + t)
        tables = [torch.from_numpy(t).pin_memory().to(rt.device, non_blocking=True) for t in cache.step_tables(range(len(sizes)))]
        views = cache.views(tables)
        segments = [Segment(i, cache.slot(i), p, [0] * t) for i, (t, p) in enumerate(sizes)]
    ctx = build_context(rt, segments, views)
    h = state["norm_in"].forward(ctx, x, None)
    args = (ctx, h) if cache is None else (ctx, h, views[0])
    delta = part.forward(*args, residual=x) if part.adds_to_residual else part.forward(*args)
    y = state["norm_out"].forward(ctx, x, delta)
    out = {"y": y, "x": x}
    if state["kind"] == "recurrence":
        out["state"] = cache.states[0].tensor
    elif state["kind"] == "latent":
        out["cache"] = cache.groups[0].tensor
    return out


def _turn_pairs(x, pos, theta):
    """x [..., T, D] (T at axis 0): entry 2i turned with entry 2i + 1."""
    D = x.shape[-1]
    inv = 1.0 / theta ** (torch.arange(0, D, 2, dtype=torch.float64, device=DEV) / D)
    a = pos.to(torch.float64).view(-1, *([1] * (x.dim() - 2)), 1) * inv
    c, s, u, v = torch.cos(a), torch.sin(a), x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2)


def _exact_latent(case, seed, z, w, h):
    H, D, R, V, r, out, at = z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"], [], 0
    for (t, p), past in zip(_portions(case), _past_rows(case, seed)):
        rows, pos = h[at:at + t], p + torch.arange(t, device=DEV)
        at += t
        q = (rows @ w["m.q"].T).view(t, H, D + R)
        ckv = rows @ w["m.dkv"].T
        c = torch.cat([past[:, :r].double(), _rms(ckv[:, :r], w["m.dkv.norm"])])
        key = torch.cat([past[:, r:].double(), _turn_pairs(ckv[:, r:], pos, 1e4)])
        k = torch.cat([(c @ w["m.uk"].T).view(-1, H, D), key[:, None, :].expand(-1, H, R)], dim=-1)
        o = _attend(torch.cat([q[..., :D], _turn_pairs(q[..., D:], pos, 1e4)], dim=-1), k, (c @ w["m.uv"].T).view(-1, H, V), p, (D + R) ** -0.5)
        out.append(o.reshape(t, H * V) @ w["m.o"].T)
    return torch.cat(out), None


def _exact_experts(case, seed, z, w, h):
    silu = torch.nn.functional.silu
    s = torch.softmax(h @ w["m.router"].T, dim=-1)
    best = s.view(len(s), z["groups"], -1).amax(-1)
    kept = torch.zeros_like(best).scatter_(1, best.topk(z["keep"], dim=-1).indices, 1.0)
    wt, idx = (s * kept.repeat_interleave(z["experts"] // z["groups"], dim=1)).topk(z["top"], dim=-1)
    out = (silu(h @ w["m.shared.gate"].T) * (h @ w["m.shared.up"].T)) @ w["m.shared.down"].T
    for k in range(z["experts"]):
        rows, col = (idx == k).nonzero(as_tuple=True)
        v = h[rows]
        out.index_add_(0, rows, wt[rows, col][:, None] * ((silu(v @ w[f"m.e{k}.gate"].T) * (v @ w[f"m.e{k}.up"].T)) @ w[f"m.e{k}.down"].T))
    return out, None


def _exact_recurrence(case, seed, z, w, h):
    H, D, V, out, at = z["heads"], z["dim"], z["vdim"], [], 0
    state = _past_state(case, seed).double()
    q = torch.nn.functional.silu(h @ w["m.q"].T).view(-1, H, D)
    f = (w["m.lower"] + (1.0 - w["m.lower"]) * torch.sigmoid(h @ w["m.f"].T + w["m.f.b"])).view(-1, H, D)
    v = (h @ w["m.v"].T).view(-1, H, V)
    for i, (t, _) in enumerate(_portions(case)):
        S = state[i]
        for j in range(at, at + t):
            S = f[j][:, :, None] * S + (1.0 - f[j])[:, :, None] * v[j][:, None, :]
            out.append(torch.einsum("hdv,hd->hv", S, q[j]))
        state[i] = S
        at += t
    return _rms(torch.stack(out), w["m.norm"]).reshape(-1, H * V) @ w["m.o"].T, state


def _exact_sublayer(case, seed):
    z, specs = _sublayer_specs(case)
    w = {k: v.double() for k, v in _make(specs, seed).items()}
    x = _normal((case["tokens"], z["width"]), 1.0, seed, 5).double()
    d, state = {"latent": _exact_latent, "experts": _exact_experts, "recurrence": _exact_recurrence}[case["kind"]](case, seed, z, w, _rms(x, w["n1"]))
    out = {"y": _rms(x + d, w["n2"]), "x": x + d}
    if case["kind"] == "recurrence":
        out["state"] = state
    elif case["kind"] == "latent":
        out["cache"] = None
    return out


def _work_sublayer(case):
    z, specs = _sublayer_specs(case)
    T, W, sizes = case["tokens"], z["width"], _portions(case)
    weights = sum(math.prod(shape) for name, shape, _ in specs if len(shape) > 1 and not name.startswith("m.e"))
    nbytes, flops = 2.0 * weights + T * W * (4 + 4 + 2), 2.0 * T * weights   # the stream in and out, the normed rows out
    if case["kind"] == "latent":
        row = z["rank"] + z["rot"]
        pairs = sum(t * p + t * (t + 1) / 2 for t, p in sizes)
        # keys and values made per head from the latents, or the latents read by all heads: scores and sums of the narrower form
        flops += 2.0 * z["heads"] * pairs * (z["dim"] + z["rot"] + z["vdim"])
        nbytes += 2.0 * row * sum(t + p for t, p in sizes)
    elif case["kind"] == "experts":
        used = min(z["experts"], T * z["top"])
        nbytes += 2.0 * used * 3 * z["ff"] * W
        flops += 2.0 * T * z["top"] * 3 * z["ff"] * W
    else:
        nbytes += 8.0 * len(sizes) * z["heads"] * z["dim"] * z["vdim"]
        flops += 4.0 * T * z["heads"] * z["dim"] * z["vdim"]
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------- what is asked of every case
def _whole(case):
    return case["kind"] in ("decode", "portion")


def prepare(case, seed):
    return _prepare_model(case, seed) if _whole(case) else _prepare_sublayer(case, seed)


def run(state):
    return _run_model(state) if _whole(state) else _run_sublayer(state)


def exact(case, seed):
    return _exact_model(case, seed) if _whole(case) else _exact_sublayer(case, seed)


def work(case):
    return _work_model(case) if _whole(case) else _work_sublayer(case)


def tolerance(case):
    """About four times the distance of this path from 64 bits (measured: 3.4e-6 in float32; 0.006 to 0.013 for the logits of whole bfloat16
    models, 0.0018 for a latent-attention sublayer, 0.0024 for a recurrence; 0.011 for the experts, where rounding the rows to bfloat16 turns
    some choices of nearly equal experts)."""
    if case.get("dtype") == "float32":
        return {"rel": 1.4e-5}
    return {"rel": {"latent": 0.007, "experts": 0.03, "recurrence": 0.01}.get(case["kind"], 0.03)}
