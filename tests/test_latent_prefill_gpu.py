"""Latent attention of prompt portions through keys and values per head, at the edges of its tiles and variants."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _g(seed):
    return torch.Generator().manual_seed(seed)


@pytest.mark.parametrize("dim,rot,vdim,rank,page", [(128, 64, 128, 512, 16), (64, 32, 64, 256, 64), (128, 0, 64, 96, 8), (64, 8, 128, 40, 128)])
@pytest.mark.parametrize("window", [None, 70])
def test_kernels_match_the_formulas(dim, rot, vdim, rank, page, window):
    """Gather, product and attention on ragged segments, with and without a window, a sink and a gate, against float64."""
    from inference_bench_b200.kernels import ops
    heads, g = 3, _g(dim + rot + page)
    segs = [(1, 0), (63, 1), (64, 64), (65, 0), (128, 63), (129, 130), (300, 7), (40, 500)]     # (tokens, cached before)
    total = sum(-(-(n + p) // page) for n, p in segs)
    pool = torch.full((1, total + 1, 1, 1, page, rank + rot), float("nan"))
    order, at, tables, rows = torch.randperm(total + 1, generator=g).tolist(), 0, [], []
    width = max(-(-(n + p) // page) for n, p in segs)
    for n, p in segs:
        pages = order[at:at + -(-(n + p) // page)]
        at += len(pages)
        r = torch.randn(n + p, rank + rot, generator=g).to(torch.bfloat16)
        rows.append(r.double())
        lowest = 0 if window is None else max(0, p - window + 1) // page    # pages before the window are gone
        tables.append([-1] * lowest + pages[lowest:] + [-1] * (width - len(pages)))
        for j, pg in enumerate(pages):
            part = r[j * page:(j + 1) * page].float()
            pool[0, pg, 0, 0, :len(part)] = part
    view = ops.KvLayerView(pool.to(torch.bfloat16).to(DEV), 0, torch.tensor(tables, dtype=torch.int32, device=DEV))
    starts = [0]
    for n, _ in segs:
        starts.append(starts[-1] + n)
    T = starts[-1]
    w = (torch.randn(heads * (dim + vdim), rank, generator=g) * rank ** -0.5).to(torch.bfloat16)
    qn, qf = torch.randn(T, heads, dim, generator=g).to(torch.bfloat16), torch.randn(T, heads, rank + rot, generator=g)
    sink, gate = torch.randn(heads, generator=g), torch.randn(2, T, heads + 2, generator=g)
    blocks, tiles = [], []
    for s, (n, p) in enumerate(segs):
        first = 0 if window is None else max(0, p - window + 1) // 64 * 64
        base = 64 * len(blocks) - first
        blocks += [(s, k) for k in range(first, n + p, 64)]
        tiles += [(starts[s] + a, min(128, n - a), p + a, base) for a in range(0, n, 128)]
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    kv, part = ops.latent_keys_values(view, i32(blocks), i32(starts), i32([p for _, p in segs]), w.to(DEV), rank, rot, status, window)
    out = torch.full((T, heads, vdim), float("nan"), dtype=torch.bfloat16, device=DEV)
    scale = 1 / math.sqrt(dim + rot)
    ops.latent_prefill(qn.to(DEV), qf.to(DEV), rank, i32(tiles), kv, part, scale, out, status, window=window, sink=sink.to(DEV), gate=(gate.to(DEV), 2))
    assert status.item() == 0
    q = torch.cat([qn.double(), qf[..., rank:].to(torch.bfloat16).double()], dim=-1)
    wd = w.double().view(-1, rank)
    for s, (n, p) in enumerate(segs):
        c = rows[s][:, :rank]
        made = (c @ wd.T).to(torch.bfloat16).double()      # keys and values are rounded once, as the product's results
        k, v = made[:, :heads * dim].view(-1, heads, dim), made[:, heads * dim:].view(-1, heads, vdim)
        k = torch.cat([k, rows[s][:, None, rank:].expand(-1, heads, rot)], dim=-1)
        sc = torch.einsum("thd,khd->htk", q[starts[s]:starts[s + 1]], k) * scale
        pos, key = p + torch.arange(n)[:, None], torch.arange(n + p)[None]
        sc = sc.masked_fill((key > pos) | ((key <= pos - window) if window else (key < 0)), -math.inf)
        sc = torch.cat([sc, sink.double()[:, None, None].expand(-1, n, 1)], dim=-1)
        ref = torch.einsum("htk,khv->thv", torch.softmax(sc, dim=-1)[..., :-1], v) * torch.sigmoid(gate.double().sum(0)[starts[s]:starts[s + 1], 2:])[..., None]
        got = out[starts[s]:starts[s + 1]].cpu().double()
        # weights and results are rounded to bfloat16 (2^-9 each), keys and values may round the other way: a few 2^-9 of the largest value
        assert (got - ref).abs().max() <= 6 * 2.0 ** -9 * v.abs().max(), (s, n, p)


@pytest.mark.parametrize("q_rank,gate,sink,window,dim,rot", [(None, False, False, None, 128, 64), (48, True, True, 100, 64, 32), (48, False, True, None, 128, 0)])
def test_a_step_of_portions_and_tokens_matches_the_other_form(q_rank, gate, sink, window, dim, rot):
    """The part on a step that holds portions of both forms beside decoded tokens, cut in two, against the form that reads the latents."""
    from inference_bench_b200.cache.manager import CacheManager
    from inference_bench_b200.config.runtime_options import RuntimeOptions
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import lib
    from inference_bench_b200.parts.latent import EXPAND_MIN_TOKENS, LatentAttention
    from inference_bench_b200.parts.standard import NoPositionEncoding, RotaryEmbedding
    from inference_bench_b200.weights.random_init import random_weights
    steps = [[90, 200, EXPAND_MIN_TOKENS - 1, 5], [1, 140, EXPAND_MIN_TOKENS, 1]]
    outs, names = {}, []
    for how in ("auto", "mma"):
        rt = Runtime(DEV, options=RuntimeOptions(latent_attention=how))
        position = RotaryEmbedding(rot, 1e4, pairing="interleaved") if rot else NoPositionEncoding()
        att = LatentAttention("a", 96, 4, dim, rot, 64, 128, (dim + rot) ** -0.5, 1e-5, position, window=window, q_rank=q_rank, gate=gate, sink=sink)
        att.bind({k: v.to(DEV) for k, v in random_weights(att.weight_specs(), 3, std=0.1).items()}, rt)
        cache = CacheManager([att.cache_need()], 16, 64, 4, 512, device=rt.device, dtype=rt.act_dtype)
        real = lib.call
        for i in range(4):
            cache.admit(i)
        got, g = [], _g(5)
        for lens in steps:
            for i, n in enumerate(lens):
                cache.extend(i, cache.length(i) + n)
            tables = [torch.from_numpy(t).to(DEV) for t in cache.step_tables(range(4))]
            ctx = build_context(rt, [Segment(i, cache.slot(i), cache.length(i), [0] * n) for i, n in enumerate(lens)], cache.views(tables))
            h = torch.randn(sum(lens), 96, generator=g).to(torch.bfloat16).to(DEV)
            lib.call = lambda name, *a: (names.append((how, name)), real(name, *a))[1]
            try:
                got.append(att.forward(ctx, h, ctx.caches[0]).sum(0))
            finally:
                lib.call = real
            for i, n in enumerate(lens):
                cache.commit(i, cache.length(i) + n)
        rt.check_status()
        outs[how] = got
    assert ("auto", "ib_latent_prefill") in names and ("auto", "ib_latent_attention_mma") in names and ("mma", "ib_latent_prefill") not in names
    for a, b in zip(outs["auto"], outs["mma"]):
        # two roundings of values and weights to bfloat16 in either form, summed over 4 heads of 64
        assert (a - b).abs().max() <= 2e-2 * b.abs().max()


@pytest.mark.parametrize("K,n,rows", [(64, 256, [0]), (128, 512, list(range(70))), (256, 64, [3, 4, 9, 63, 64, 65, 130, 199]), (40, 33, list(range(199, 60, -1)))])
def test_the_maps_of_a_list_of_rows(K, n, rows):
    """Rows of a list give the bits that they have among all rows; the others are not read (they are NaN) and not written."""
    from inference_bench_b200.kernels import ops
    T, heads, g = 200, 3, _g(K + n)
    x = torch.randn(T, heads, K, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(heads, n, K, generator=g).to(torch.bfloat16).to(DEV)
    gate = (torch.randn(2, T, heads + 1, generator=g).to(DEV), 1)
    whole = torch.empty(T, heads, n + 8, device=DEV)
    ops.gemm_heads(x, w, whole, n, tensor_cores=True, gate=gate)
    at = torch.tensor(rows, device=DEV)
    some, out = torch.full_like(x, float("nan")), torch.full((T, heads, n + 8), 7.0, device=DEV)
    some[at] = x[at]
    ops.gemm_heads(some, w, out, n, tensor_cores=True, gate=gate, rows=at.int())
    assert torch.equal(out[at, :, :n], whole[at, :, :n])
    rest = torch.ones(T, dtype=torch.bool, device=DEV)
    rest[at] = False
    assert (out[rest] == 7.0).all() and (out[..., n:] == 7.0).all()
