"""Regrouping pairs by expert and gathering rows at the edges of what a thread keeps and a warp copies."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,top,E,tile", [(1, 1, 1, 16), (3, 5, 31, 32), (1023, 1, 32, 64), (1025, 1, 33, 128), (2730, 6, 64, 128), (16384, 1, 65, 128), (16385, 1, 2, 256),
                                          (7000, 6, 300, 128)])
def test_sort(T, top, E, tile):
    from inference_bench_b200.kernels import ops
    g = torch.Generator().manual_seed(T + E)
    idx = torch.randint(0, E, (T, top), generator=g, dtype=torch.int32)
    i32 = lambda n: torch.full((n,), -7, dtype=torch.int32, device=DEV)
    offsets, tiles, row, token = i32(E + 1), i32(E + 1), i32(T * top), i32(T * top)
    ops.moe_sort(idx.to(DEV), E, offsets, tiles, row, token, tile_rows=tile)
    counts = torch.bincount(idx.flatten().long(), minlength=E)
    assert offsets.cpu().tolist() == [0] + counts.cumsum(0).tolist()
    assert tiles.cpu().tolist() == [0] + ((counts + tile - 1) // tile).cumsum(0).tolist()
    row = row.cpu().long()
    assert torch.equal(row.sort().values, torch.arange(T * top))
    assert torch.equal(token.cpu()[row], torch.arange(T * top, dtype=torch.int32) // top)
    group = torch.empty(T * top, dtype=torch.int32)
    group[row] = idx.flatten()
    assert torch.equal(group.sort(stable=True).values, group)


@pytest.mark.parametrize("R,K", [(1, 8), (7, 1016), (8, 1024), (9, 1032), (100, 8200), (65, 16400)])
def test_gather(R, K):
    from inference_bench_b200.kernels import ops
    x = torch.randn((33, K), device=DEV).to(torch.bfloat16)
    src = torch.randint(0, 33, (R,), dtype=torch.int32, device=DEV)
    out = torch.full((R + 1, K), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.gather_rows(x, src, out[:R])
    assert torch.equal(out[:R], x[src.long()]) and (out[R] == 7).all()
