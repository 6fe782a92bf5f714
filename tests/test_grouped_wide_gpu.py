"""Experts' products on CTA pairs in token tiles of 256 rows, loaded and multiplied only as far as an expert's rows go (csrc/gemm_tcgen05_2cta.cu)."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import DEV, _g

pytestmark = pytest.mark.gpu


# experts without rows (the first and the last among them), with one, around every step of 16 and 32 rows and around one and two tiles; matrices whose last
# block of rows is partly there, the smallest, and an inner size with a remainder; the last group's up rows end at the buffer's end
@pytest.mark.parametrize("counts,N,K", [([0, 1, 15, 16, 17, 0], 16, 8), ([31, 32, 33, 63, 64, 65, 95], 272, 72), ([127, 129, 0, 255, 256, 257, 1], 144, 200), ([513, 0, 0, 480, 3], 400, 64),
                                        ([70] * 40, 128, 136), ([0, 0, 300], 1408, 2048)])
def test_products_of_regrouped_rows(counts, N, K):
    from inference_bench_b200.kernels import gemm_tcgen05 as G, ops
    status, E, R = torch.zeros(1, dtype=torch.int32, device=DEV), len(counts), sum(counts)
    table = lambda per: torch.tensor([0] + torch.tensor(per).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    offsets, tiles = table(counts), table([-(-c // G.PAIR_WIDE_TILE) for c in counts])
    x = (torch.randn((R, K), generator=_g(R)) * 0.5).to(torch.bfloat16).to(DEV)
    w = (torch.randn((E, 2 * N, K), generator=_g(E)) * 0.5).to(torch.bfloat16).to(DEV)
    limits, slope = torch.linspace(0.5, 3.0, E), 1.7
    parts = [x[a:b].double() @ w[e].double().T for e, (a, b) in enumerate(zip(offsets.tolist(), offsets.tolist()[1:]))]
    whole, own = torch.cat(parts), torch.repeat_interleave(limits, torch.tensor(counts)).double()[:, None].to(DEV)
    bound = K * 2.0 ** -24 * max(float((x[a:b].double().abs() @ w[e].double().abs().T).max()) for e, (a, b) in enumerate(zip(offsets.tolist(), offsets.tolist()[1:])) if b > a)
    guard = 64   # rows behind the last expert's that must stay as they are
    out = torch.full((R + guard, 2 * N), 7.0, device=DEV)
    G.gemm_grouped(x, w, out[:R], 256, offsets, tiles, status, pair=True)
    assert ((out[:R].double() - whole).abs() <= bound).all() and (out[R:] == 7.0).all()
    act = torch.full((R + guard, 2 * N), 7.0, device=DEV, dtype=torch.bfloat16)
    G.gemm_grouped_relu2(x, w, act[:R], 256, offsets, tiles, status, pair=True)
    want = whole.clamp(min=0) ** 2
    assert ((act[:R].double() - want).abs() <= 2.0 ** -8 * want + 3 * bound * whole.abs().max()).all() and (act[R:] == 7.0).all()
    gate, up = whole[:, :N], whole[:, N:]
    for clamp in (None, ops.Clamp(limits.float().to(DEV), slope)):
        g, u = (gate, up) if clamp is None else (torch.minimum(gate, own), torch.minimum(torch.maximum(up, -own), own))
        want = g * torch.sigmoid(g * (1.0 if clamp is None else slope)) * (u if clamp is None else u + 1.0)
        act = torch.full((R + guard, N), 7.0, device=DEV, dtype=torch.bfloat16)
        G.gemm_grouped_swiglu(x, w, act[:R], 256, offsets, tiles, status, clamp=clamp, pair=True)
        # one rounding to bfloat16, approximate exponential and division (a few 2^-22), and the sums' own error through a function of slope below 2
        assert ((act[:R].double() - want).abs() <= 2.0 ** -8 * want.abs() + 4 * bound * (1 + gate.abs().max() + up.abs().max())).all() and (act[R:] == 7.0).all()
        narrow = torch.empty((R, N), device=DEV, dtype=torch.bfloat16)
        G.gemm_grouped_swiglu(x, w, narrow, 128, offsets, table([-(-c // 128) for c in counts]), status, clamp=clamp, pair=True)
        assert torch.equal(narrow, act[:R])   # the same sums in the same order
    assert int(status[0]) == 0


def test_the_tile_is_chosen_by_sizes():
    from inference_bench_b200.kernels import gemm_tcgen05 as G
    assert [G.grouped_pairs(r, 64, 1408) for r in (64 * 31, 64 * 32, 64 * 128)] == [False, True, True]
    assert [G.grouped_pairs(r, 4, 256) for r in (4 * 127, 4 * 128)] == [False, True] and not G.grouped_pairs(1 << 20, 257, 1408)
    assert G.pair_tile(12288, 64, 1408) == 256 and G.pair_tile(12288, 64, 1400) == 128 and G.pair_tile(12288, 64, 1400, gated=False) == 256
    assert G.pair_tile(16 * 512, 16, 1024) == 128 and G.pair_tile(16 * 256, 16, 1024) == 256


def test_the_tile_of_small_and_large_shares():
    from inference_bench_b200.kernels import gemm_tcgen05 as G
    of = lambda avg, n, inter: G.pair_tile(avg * n, n, inter)
    assert [of(a, 128, 1536) for a in (32, 111, 112, 256, 257, 300, 512, 700)] == [128, 128, 256, 256, 128, 128, 128, 128]
    assert [of(a, 64, 1408) for a in (32, 192, 257)] == [256, 256, 128]   # (5.5 blocks of 256 gate rows are 6)
    assert [of(64, 16, 1024), of(64, 32, 1024), of(64, 32, 2880)] == [256, 128, 128]
