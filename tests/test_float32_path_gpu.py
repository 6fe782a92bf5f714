"""The float32 path's product and prompt attention at the edges of their tiles."""
from __future__ import annotations

import math

import pytest
import torch

from test_kernels_gpu import DEV, _attention_case, _g, status  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


# tiles of 16 x 16, 16 x 64, 32 x 32, 32 x 64 and 64 x 64, with remainders in every size, inner sizes that no vector load takes, and the smallest
@pytest.mark.parametrize("T,N,K", [(1, 1, 1), (3, 17, 5), (16, 9473, 68), (15, 100, 200), (17, 16, 64), (100, 1531, 130), (129, 4799, 36), (333, 2050, 260), (640, 4100, 72), (70, 130, 41)])
@pytest.mark.parametrize("x_dtype,w_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16)])
def test_product_at_tile_edges(T, N, K, x_dtype, w_dtype):
    from inference_bench_b200.kernels import ops
    g = _g(T + N + K)
    x, w = torch.randn(T, K, generator=g).to(x_dtype).to(DEV), torch.randn(N, K, generator=g).to(w_dtype).to(DEV)
    out = torch.full((T, N), float("nan"), device=DEV)
    ops.gemm_simt(x, w, out)
    xd, wd = x.double(), w.double()
    # a chain of n FMAs is off by at most n eps times the sum of magnitudes; the longest of the four chains has ceil(K / 64) * 16 terms, two additions follow
    bound = (-(-K // 64) * 16 + 3) * 2.0 ** -24 * (xd.abs() @ wd.abs().T)
    assert ((out.double() - xd @ wd.T).abs() <= bound).all()
    # a row does not depend on how many others there are
    alone = torch.empty(1, N, device=DEV)
    ops.gemm_simt(x[-1:].contiguous(), w, alone)
    assert torch.equal(alone[0], out[-1])


# the tiles that only some sizes are given (csrc/gemm_simt.cu, FORMS): 16 x 64 above 16 rows, 48 x 64, 64 x 64, 40 x 128, 48 x 128, 56 x 128, 64 x 96 and
# 64 x 128, with remainders in rows and columns and inner sizes with and without vector loads
@pytest.mark.parametrize("T,N,K", [(33, 2563, 33), (129, 2050, 72), (193, 2050, 65), (33, 9473, 36), (513, 1540, 68), (193, 4099, 41), (41, 9473, 130), (289, 3077, 64)])
@pytest.mark.parametrize("x_dtype,w_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_product_at_the_edges_of_wide_tiles(T, N, K, x_dtype, w_dtype):
    test_product_at_tile_edges(T, N, K, x_dtype, w_dtype)


@pytest.mark.parametrize("hd,heads,kvh,page", [(128, 4, 2, 16), (64, 6, 1, 8), (128, 3, 3, 64)])
@pytest.mark.parametrize("variant", ["plain", "window", "window_keep", "chunk", "cap_sink", "tail"])
def test_prompt_attention_matches_the_row_kernel(status, hd, heads, kvh, page, variant):  # noqa: F811
    """Portions around the tiles' 64 rows and 64 keys beside decoded tokens, against the kernel that takes a row a warp and (plain, window) the
    plain reference; every portion alone gives the same bits."""
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import attention, ops
    window = 45 if variant.startswith("window") else None
    shapes = [(300, 300), (200, 70), (97, 1), (64, 64), (65, 65), (33, 2), (129, 128), (31, 31)]
    q, view, pos, seg, ref, _ = _attention_case(torch.float32, heads, kvh, hd, page, window, shapes, 21)
    T, scale, g = q.shape[0], 1 / math.sqrt(hd), _g(22)
    kw = {"plain": {}, "window": {}, "window_keep": dict(keep_first=37), "chunk": dict(chunk=50),
          "cap_sink": dict(softcap=2.0, sink=True, sink_values=torch.randn(heads, generator=g).to(DEV)),
          "tail": dict(sink=True, out_scale=0.5, gate=(torch.randn(2, T, heads + 3, generator=g).to(DEV), 3))}[variant]
    rt = Runtime(DEV, "float32")

    def run(rows, segments):
        ctx = build_context(rt, segments)
        sub = ops.KvLayerView(view.pool, view.entry, view.block_table[[s.request for s in segments]].contiguous())
        more = dict(kw, gate=(kw["gate"][0][:, rows].contiguous(), 3)) if "gate" in kw else kw
        wide = torch.full((ctx.n_tokens, heads * hd + 8), 7.0, device=DEV)
        attention.paged_attention(ctx, q[rows].contiguous(), sub, heads, window, scale, out=wide, **more)
        assert (wide[:, heads * hd:] == 7.0).all()
        return wide[:, :heads * hd]

    segs = [Segment(i, i, L - n, [0] * n) for i, (L, n) in enumerate(shapes)]
    out = run(slice(0, T), segs)
    rt.check_status()
    want = torch.empty_like(q)
    ops.attention_generic(q, view, pos, seg, window, scale, want, heads, status, **kw)
    # both sum up to 300 weighted values in float32: a few tens of roundings of values up to the largest output
    assert (out - want).abs().max() <= 64 * 2.0 ** -24 * want.abs().max().clamp(min=1.0)
    if variant in ("plain", "window"):
        assert (out.cpu().double() - ref).abs().max() <= 1e-5 * ref.abs().max()
    at = 0
    for s, (_, n) in zip(segs, shapes):
        assert torch.equal(run(slice(at, at + n), [s]), out[at:at + n])
        at += n


@pytest.mark.parametrize("hd,heads,kvh,page", [(128, 4, 2, 16), (64, 6, 1, 8)])
@pytest.mark.parametrize("variant", ["plain", "window", "window_keep", "chunk", "cap_sink", "gate_sink"])
def test_prompt_attention_gives_the_bits_of_the_row_kernel(hd, heads, kvh, page, variant):
    """A position's result does not depend on the kernel that computes it: portions whose rows start anywhere in a tile, with windows and blocks
    that begin anywhere in a run of 32 keys."""
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import attention, lib, ops
    window = 77 if variant.startswith("window") else None
    shapes = [(300, 300), (200, 70), (161, 33), (64, 64), (65, 63), (33, 2), (257, 128)]
    q, view, pos, seg, _, _ = _attention_case(torch.float32, heads, kvh, hd, page, window, shapes, 23)
    T, scale, g = q.shape[0], 1 / math.sqrt(hd), _g(24)
    kw = {"plain": {}, "window": {}, "window_keep": dict(keep_first=37), "chunk": dict(chunk=50), "cap_sink": dict(softcap=2.0, sink=True, sink_values=torch.randn(heads, generator=g).to(DEV)),
          "gate_sink": dict(sink=True, out_scale=0.3, gate=(torch.randn(3, T, heads + 3, generator=g).to(DEV), 2))}[variant]
    rt = Runtime(DEV, "float32")
    names, real = [], lib.call
    lib.call = lambda name, *a: (names.append(name), real(name, *a))[1]
    try:
        out = attention.paged_attention(build_context(rt, [Segment(i, i, L - n, [0] * n) for i, (L, n) in enumerate(shapes)]), q, view, heads, window, scale, **kw)
    finally:
        lib.call = real
    want = torch.empty_like(q)
    ops.attention_generic(q, view, pos, seg, window, scale, want, heads, rt.status, **kw)
    rt.check_status()
    assert names == ["ib_attention_prompt_f32"] and torch.equal(out, want)


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("windows", [(0, 0, 0), (1, 0, 1)])
def test_logits_do_not_depend_on_how_a_prompt_is_cut(head_dim, windows):
    """A prompt in one portion, with its last token alone, in odd pieces, and beside others: the same bits, in the cache too."""
    from inference_bench_b200.engine.step import StepEntry
    from test_repeat_gpu import _runner
    tokens, outs = torch.randint(0, 333, (211,), generator=_g(3)).tolist(), []
    for cuts, other in (([211], 0), ([210, 1], 0), ([1, 97, 64, 1, 48], 0), ([64, 130, 17], 9)):
        r, at = _runner("float32", head_dim, windows, 16), 0
        r.cache.admit(0), r.cache.admit(1)
        for n in cuts:
            entries = [StepEntry(1, [7 + n] * other, [])] * (other > 0) + [StepEntry(0, tokens[at:at + n], [n - 1])]
            logits = r.step(entries)
            at += n
        rows = [[(gr.tensor[:, p].clone(), min(16, 211 - 16 * i)) for i, p in enumerate(r.cache.table(g, 0)[:14].tolist()) if p >= 0] for g, gr in enumerate(r.cache.groups)]
        outs.append((logits.clone(), [[t[..., :n, :] for t, n in row] for row in rows]))
    for logits, rows in outs[1:]:
        assert torch.equal(logits, outs[0][0])
        for a, b in zip(rows, outs[0][1]):
            assert len(a) == len(b) > 0 and all(torch.equal(u, v) for u, v in zip(a, b))
