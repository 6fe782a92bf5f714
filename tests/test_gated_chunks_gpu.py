"""The gated recurrence's chunks as products (csrc/gated_recurrence.cu, gated_chunk_kernel) against the plain recurrence."""
from __future__ import annotations

import pytest
import torch

import plain_busadra as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# around the chunk's 64 tokens and its blocks of sixteen; heads and value columns that end inside the kernel's 128, at it and in a second block of columns
@pytest.mark.parametrize("lens", [[65], [80, 64], [127, 1, 129], [192, 97], [2048]])
@pytest.mark.parametrize("heads,D,V", [(2, 128, 128), (3, 65, 66), (1, 100, 131), (2, 72, 260)])
@pytest.mark.parametrize("gates", ["open", "closing"])
def test_against_the_plain_recurrence(lens, heads, D, V, gates):
    """closing: floors of zero and gates down to e^-40 a token, where a quotient of running products would be 0 / 0."""
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import ops
    from inference_bench_b200.parts.recurrent import GatedLinearRecurrence
    if sum(lens) > 500 and D != 128:
        lens = [300]
    g, T, R = torch.Generator().manual_seed(D + V + sum(lens)), sum(lens), heads * (2 * D + V)
    proj = torch.randn((2, T, R), generator=g)
    f_bias, lower = torch.randn((heads * D,), generator=g), torch.rand((heads * D,), generator=g) * 0.9
    lower[::3] = 0.995
    if gates == "closing":
        f_bias = f_bias * 8 - 16
        lower[1::3] = 0.0
    state = torch.randn((len(lens) + 1, heads, D, V), generator=g)
    ctx = build_context(Runtime(DEV, "float32"), [Segment(i, i + 1, 0, [0] * n) for i, n in enumerate(lens)])
    short, long_segs, chunks = GatedLinearRecurrence._cut(ctx)
    got, out = state.to(DEV), torch.full((T, heads, V), float("nan"), device=DEV)
    dev = lambda t: t.to(DEV)
    ops.gated_recurrence(dev(proj), dev(f_bias), dev(lower), got, ctx.seg_start, ctx.seg_slot, len(lens), out, heads, D, V, seg_list=short, long_segs=long_segs, chunks=chunks)
    z, lo, at = proj.double().sum(0), lower.double().view(heads, D), 0
    q = P.silu(z[:, :heads * D]).view(T, heads, D)
    f = lo + (1 - lo) * torch.sigmoid(z[:, heads * D:2 * heads * D] + f_bias.double()).view(T, heads, D)
    v = z[:, 2 * heads * D:].view(T, heads, V)
    for i, n in enumerate(lens):
        want, last = P.recurrence_core(q[at:at + n], f[at:at + n], v[at:at + n], state[i + 1])
        # q, f and v come from float32 sums (a few 2^-24 of them); an output is a sum of D products with a state of at most a few hundred such terms
        tol = 2e-5 * max(1.0, want.abs().max().item())
        assert (out[at:at + n].cpu().double() - want).abs().max().item() < tol
        assert (got[i + 1].cpu().double() - last).abs().max().item() < 2e-5 * max(1.0, last.abs().max().item())
        at += n
    assert torch.equal(got[0].cpu(), state[0])


def test_a_token_sees_no_later_one():
    """An infinite value and a NaN gate reach the tokens behind them only."""
    from inference_bench_b200.engine.context import Segment, build_context
    from inference_bench_b200.engine.runtime import Runtime
    from inference_bench_b200.kernels import ops
    from inference_bench_b200.parts.recurrent import GatedLinearRecurrence
    heads, D, V, T = 2, 128, 128, 140
    g = torch.Generator().manual_seed(1)
    clean = torch.randn((1, T, heads * (2 * D + V)), generator=g)
    bias, lower = torch.randn((heads * D,), generator=g).to(DEV), torch.rand((heads * D,), generator=g).to(DEV)
    ctx = build_context(Runtime(DEV, "float32"), [Segment(0, 0, 0, [0] * T)])
    cut = GatedLinearRecurrence._cut(ctx)

    def run(proj):
        out = torch.empty((T, heads, V), device=DEV)
        ops.gated_recurrence(proj.to(DEV), bias, lower, torch.zeros((1, heads, D, V), device=DEV), ctx.seg_start, ctx.seg_slot, 1, out, heads, D, V, seg_list=cut[0], long_segs=cut[1], chunks=cut[2])
        return out
    want = run(clean)
    for token, column in ((70, 2 * heads * D + 5), (21, heads * D + 7), (3, 2 * heads * D)):
        bad = clean.clone()
        bad[0, token, column] = float("inf") if column >= 2 * heads * D else float("nan")
        got = run(bad)
        assert torch.equal(got[:token], want[:token]) and not torch.isfinite(got[token:]).all()
