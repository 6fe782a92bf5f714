"""Prompt portions whose keys are cut into slices over a thread-block cluster: every number of slices, slices without keys (a segment much shorter than the
longest, rows that see none of a slice), windows, kept positions, sinks and gates, page sizes on both sides of a tile."""
from __future__ import annotations

import math

import pytest
import torch
from test_kernels_gpu import _attention_case

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _slices(heads, shapes, window=None, keep=0):
    """The number of slices on a device of 148 SMs."""
    from inference_bench_b200.kernels import attention, lib
    starts = [sum(n for _, n in shapes[:i]) for i in range(len(shapes))]
    _, _, seg, _, keys = attention.work_lists([n for _, n in shapes], starts, [L - n for L, n in shapes])
    return lib.load().ib_attention_prefill_slices(heads, len(seg), keys, window or 0, keep, 148)


@pytest.mark.parametrize("hd,heads,kvh,page,shapes,slices", [
    (128, 4, 2, 64, [(1100, 61)], 8),                       # 8 slices of 18 tiles, one query tile that is half full
    (64, 6, 3, 8, [(1025, 128), (70, 2), (3, 3)], 8),       # 8 slices: segments of 17, 2 and 1 key tiles; eight pages a tile
    (128, 8, 4, 16, [(700, 100), (641, 129)], 4),           # 4 slices of 11 tiles, a query tile of one row
    (128, 32, 8, 192, [(1300, 256), (130, 130)], 2),        # 2 slices at two CTAs an SM: 128 CTAs, tiles of causal keys only beside long ones
    (64, 2, 1, 128, [(4500, 2), (2500, 300)], 8),
])
@pytest.mark.parametrize("window,keep", [(None, 0), (1000, 0), (1030, 70)])
def test_sliced_portions(hd, heads, kvh, page, shapes, slices, window, keep):
    assert _slices(heads, shapes) == slices and _slices(heads, shapes, window, keep) > 1
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import attention, ops
    q, view, pos, seg, ref, _ = _attention_case(torch.bfloat16, heads, kvh, hd, page, window, shapes, 31, needle=True)
    rt = Runtime(DEV)
    ctx = build_context(rt, [Segment(i, i, L - n, [0] * n) for i, (L, n) in enumerate(shapes)])
    scale = 1 / math.sqrt(hd)
    out = attention.paged_attention(ctx, q, view, heads, window, scale, keep_first=keep)
    again = attention.paged_attention(ctx, q, view, heads, window, scale, keep_first=keep)
    rt.check_status()
    assert torch.equal(out, again)
    other = torch.empty_like(out)
    ops.attention_generic(q, view, pos, seg, window, scale, other, heads, rt.status, keep_first=keep)
    # P is rounded to bfloat16 (2^-9 of each weight) and so is the output, on both sides
    top = ref.abs().max()
    assert (out.double() - other.double()).abs().max() <= 2e-2 * top
    if not keep:
        assert (out.cpu().double() - ref).abs().max() <= 1.5e-2 * top
    sinks, gate = torch.randn(heads, device=DEV), torch.randn((2, q.shape[0], heads), device=DEV)
    kw = dict(softcap=20.0, sink=True, sink_values=sinks, gate=(gate, 0), out_scale=0.5, keep_first=keep)
    out = attention.paged_attention(ctx, q, view, heads, window, scale, **kw)
    kw["gate"] = (gate, 0)
    ops.attention_generic(q, view, pos, seg, window, scale, other, heads, rt.status, **kw)
    rt.check_status()
    assert (out.double() - other.double()).abs().max() <= 2e-2 * top


@pytest.mark.parametrize("hd,heads,kvh,page,shape,slices", [(128, 4, 2, 64, (1100, 61), 8), (64, 8, 4, 16, (700, 100), 4), (128, 32, 8, 64, (1300, 300), 2)])
def test_what_is_not_finite_stays_so(hd, heads, kvh, page, shape, slices):
    """A query row of NaN, a key that gives infinite scores, a value that is infinite: the rows that see them are not finite, the others keep their bits."""
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import attention
    from inference_bench_b200.kernels.ops import KvLayerView
    L, n = shape
    assert _slices(heads, [shape]) == slices
    rt, pages = Runtime(DEV), -(-L // page)
    g = torch.Generator().manual_seed(hd)
    pool = torch.randn((1, pages, 2, kvh, page, hd), generator=g).to(torch.bfloat16)
    q = torch.randn((n, heads * hd), generator=g).to(torch.bfloat16)
    table = torch.arange(pages, dtype=torch.int32, device=DEV)[None]
    ctx = build_context(rt, [Segment(0, 0, L - n, [0] * n)])
    run = lambda q, pool: attention.paged_attention(ctx, q.to(DEV), KvLayerView(pool.to(DEV), 0, table), heads, None, 1 / math.sqrt(hd)).view(n, heads, hd).cpu()
    clean = run(q, pool)
    assert torch.isfinite(clean).all()
    bad = q.clone()
    bad[7, :hd] = float("nan")   # a row of the first head
    got = run(bad, pool)
    assert torch.isnan(got[7, 0]).all()
    got[7, 0] = clean[7, 0]
    assert torch.equal(got, clean)
    group, key = heads // kvh, L - n // 2   # seen by the rows behind the middle only, in the last slice
    for at in (3, key):   # (a key in the first slice, and that one)
        bad = pool.clone()
        bad[0, at // page, 0, 0, at % page, 5] = float("inf")   # scores of plus or minus infinity
        got, sees = run(q, bad), torch.arange(L - n, L) >= at
        plus = (q.view(n, heads, hd)[:, :group, 5].float() > 0) & sees[:, None]
        assert torch.isnan(got[:, :group][plus]).all() and torch.equal(got[:, group:], clean[:, group:])
        assert torch.isfinite(got[:, :group][~plus & sees[:, None]]).all()
        bad = pool.clone()
        bad[0, at // page, 1, 0, at % page, 9] = float("inf")
        got = run(q, bad)
        assert not torch.isfinite(got[sees][:, :group, 9]).any()
        same = [c for c in range(hd) if c != 9]
        assert torch.equal(got[:, :group][..., same], clean[:, :group][..., same]) and torch.equal(got[:, group:], clean[:, group:])
