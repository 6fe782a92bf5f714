"""The experts' products on CTA pairs at the edges of their tiles: groups that are empty, a row short of a tile, a tile, a row over; matrices
whose rows end inside a block of 256 or 512; reductions that end inside a k-tile."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
COUNTS = {"edges": [0, 1, 127, 0, 128, 129, 300, 0], "one": [200], "many": [(7 * e) % 5 for e in range(256)]}


@pytest.mark.parametrize("counts", COUNTS, ids=str)
@pytest.mark.parametrize("N,K", [(8, 8), (264, 72), (520, 200), (136, 1024)])
def test_products_of_regrouped_rows(counts, N, K):
    """Against float64 on the same operands. A sum of K products of bfloat16 numbers in float32 is off by at most K 2^-24 times the sum of
    their sizes (tighter where it matters: K <= 1,024 gives 2^-14 of it); a bfloat16 result adds 2^-8 of itself, the fast exponential and
    division 2^-20 of their value; silu(g) u moves by at most 1.1 |dg| |u| + |g| |du|."""
    from inference_bench_b200.kernels import gemm_tcgen05 as G, ops
    counts, status = COUNTS[counts], torch.zeros(1, dtype=torch.int32, device=DEV)
    E, R = len(counts), sum(counts)
    if E > 8 and N * K > 30_000:
        N, K = 24, 72
    g = torch.Generator().manual_seed(N + K + R)
    x = torch.randn((R, K), generator=g).to(DEV, torch.bfloat16)
    w = (torch.randn((E, 2 * N, K), generator=g) / K ** 0.5).to(DEV, torch.bfloat16)
    group = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))
    table = lambda per: torch.tensor([0] + torch.tensor(per).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    offsets, tiles = table(counts), table([-(-c // G.PAIR_TILE) for c in counts])
    want, size = torch.empty((R, 2 * N), dtype=torch.float64), torch.empty((R, 2 * N), dtype=torch.float64)
    for e in range(E):
        rows = group == e
        xe, we = x[rows.to(DEV)].cpu().double(), w[e].cpu().double()
        want[rows], size[rows] = xe @ we.T, xe.abs() @ we.abs().T
    err = K * 2.0 ** -24 * size
    out = torch.full((R, 2 * N), 7.0, device=DEV)
    G.gemm_grouped(x, w, out, G.PAIR_TILE, offsets, tiles, status, pair=True)
    assert ((out.cpu().double() - want).abs() <= err).all()
    act = torch.full((R, 2 * N), 7.0, device=DEV, dtype=torch.bfloat16)
    G.gemm_grouped_relu2(x, w, act, G.PAIR_TILE, offsets, tiles, status, pair=True)
    square = want.clamp(min=0) ** 2
    assert ((act.cpu().double() - square).abs() <= 2.0 ** -8 * square + 2.1 * err * want.abs() + err ** 2 + 2.0 ** -133).all()
    gate, up, dg, du = want[:, :N], want[:, N:], err[:, :N], err[:, N:]
    glu = gate * torch.sigmoid(gate) * up
    act = torch.full((R, N), 7.0, device=DEV, dtype=torch.bfloat16)
    G.gemm_grouped_swiglu(x, w, act, G.PAIR_TILE, offsets, tiles, status, pair=True)
    assert ((act.cpu().double() - glu).abs() <= (2.0 ** -8 + 2.0 ** -18) * glu.abs() + 1.2 * (dg * up.abs() + du * gate.abs() + dg * du) + 2.0 ** -133).all()
    limits = 0.3 + torch.arange(E) % 3
    lim, slope = limits[group].double()[:, None], 1.7
    cg, cu = torch.minimum(gate, lim), torch.maximum(torch.minimum(up, lim), -lim) + 1
    glu = cg * torch.sigmoid(slope * cg) * cu
    G.gemm_grouped_swiglu(x, w, act, G.PAIR_TILE, offsets, tiles, status, clamp=ops.Clamp(limits.float().to(DEV), slope), pair=True)
    near = 2.0 ** -23 * lim     # the limits in float32
    assert ((act.cpu().double() - glu).abs() <= (2.0 ** -8 + 2.0 ** -18) * glu.abs() + 1.2 * ((dg + near) * cu.abs() + (du + near) * cg.abs() + dg * du) + 2.0 ** -24).all()
    assert status.item() == 0


def test_other_tiles_are_refused():
    from inference_bench_b200.kernels import gemm_tcgen05 as G, lib as L
    x, w, out = torch.zeros((4, 8), device=DEV, dtype=torch.bfloat16), torch.zeros((1, 8, 8), device=DEV, dtype=torch.bfloat16), torch.zeros((4, 8), device=DEV)
    t = torch.tensor([0, 4], dtype=torch.int32, device=DEV)
    with pytest.raises(L.KernelError):
        G.gemm_grouped(x, w, out, 64, t, t, torch.zeros(1, dtype=torch.int32, device=DEV), pair=True)
