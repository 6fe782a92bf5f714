"""The recurrence's chunk walk with four columns a thread: sizes around its tiles, against the token-by-token walk in float64."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# enough chunks for the form with four columns (2 x 148 CTAs), and one case below that; state sizes that end inside a group of rows or columns
@pytest.mark.parametrize("heads,D,V,T", [(16, 128, 128, 700), (12, 128, 100, 900), (20, 100, 64, 1000), (40, 36, 65, 300), (24, 7, 33, 900), (3, 128, 128, 130)])
@pytest.mark.parametrize("parts", [1, 3])
def test_chunk_walk(heads, D, V, T, parts):
    from inference_bench_b200.kernels import ops
    g = torch.Generator().manual_seed(heads + D + V)
    R = 2 * heads * D + heads * V
    proj = torch.randn(parts, T, R, generator=g) / parts ** 0.5
    bias, lower = torch.randn(heads * D, generator=g), torch.rand(heads * D, generator=g) * 0.9
    state = torch.randn(3, heads, D, V, generator=g)
    C = ops.RECURRENCE_CHUNK
    chunks = [(t, min(C, T - t)) for t in range(0, T, C)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    st, out = state.to(DEV), torch.full((T, heads, V), float("nan"), device=DEV)
    ops.gated_recurrence(proj.to(DEV), bias.to(DEV), lower.to(DEV), st, i32([0, T]), i32([1]), 1, out, heads, D, V, seg_list=i32([]), long_segs=i32([[0, 0, len(chunks)]]),
                         chunks=i32(chunks))
    z = proj.double().sum(0)
    q, f, v = (z[:, a:b].view(T, heads, -1) for a, b in ((0, heads * D), (heads * D, 2 * heads * D), (2 * heads * D, R)))
    q = torch.nn.functional.silu(q).to(DEV)
    lo = lower.double().view(heads, D)
    f = (lo + (1 - lo) * torch.sigmoid(f + bias.double().view(heads, D))).to(DEV)
    S, v, ref = state[1].double().to(DEV), v.to(DEV), []
    for t in range(T):
        S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None, :]
        ref.append(torch.einsum("hdv,hd->hv", S, q[t]))
    ref = torch.stack(ref)
    # float32 sums of D products of values around one, over states that forget: a few hundred roundings at most
    assert (out.double() - ref).abs().max() <= 512 * 2.0 ** -24 * ref.abs().max()
    assert (st[1].double() - S).abs().max() <= 512 * 2.0 ** -24 * S.abs().max()
    assert torch.equal(st[0].cpu(), state[0]) and torch.equal(st[2].cpu(), state[2])
