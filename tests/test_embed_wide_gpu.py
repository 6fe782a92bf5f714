"""The embedding with 16-byte accesses: rows of one chunk, of fewer and more than a thread's four, and rows that only the narrow form takes."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [4, 8, 12, 1000, 1024, 4096, 5120, 8200])
def test_embed(dtype, H):
    from inference_bench_b200.kernels import ops
    table = torch.randn(50, H, generator=torch.Generator().manual_seed(H)).to(dtype).to(DEV)
    toks = torch.tensor([0, 49, 7, 7, 31], dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x = torch.full((5, H), float("nan"), device=DEV)
    ops.embed(table, toks, x, status)
    assert torch.equal(x, table.float()[toks.long()]) and status.item() == 0
    odd = table.view(-1)[1:1 + 49 * H].view(49, H)      # rows that start off 16 bytes
    ops.embed(odd, toks.clamp(max=48), x, status)
    assert torch.equal(x, odd.float()[toks.clamp(max=48).long()])
    ops.embed(table, torch.tensor([3, 50, -1, 2, 1], dtype=torch.int32, device=DEV), x, status)
    assert status.item() == 2 and torch.equal(x[1], table[0].float())
