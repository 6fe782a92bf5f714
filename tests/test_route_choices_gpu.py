"""The router's choices where many scores are alike (zeros of both signs among them), where fewer experts are eligible than are chosen, beyond the 32
choices that a warp holds, and over more partial sums than are requested together."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,E,groups,keep,top,P", [(1, 4, 1, 1, 1, 1), (5, 33, 1, 1, 31, 2), (130, 64, 1, 1, 32, 8), (67, 200, 1, 1, 33, 9), (9, 300, 1, 1, 65, 17),
                                                   (70, 64, 8, 3, 6, 10), (66, 32, 8, 1, 6, 1)])
def test_choices(T, E, groups, keep, top, P):
    from inference_bench_b200.kernels import ops
    g = torch.Generator().manual_seed(E + top)
    parts = torch.randint(-3, 4, (P, T, E), generator=g).float()   # whole numbers: every sum is exact, and many are alike
    logits = parts.sum(0)
    parts[0, 0] = torch.where(torch.arange(E) % 2 == 0, -0.0, 0.0)   # token 0: zeros of both signs are alike
    parts[1:, 0] = -0.0
    logits[0] = 0.0
    idx = torch.full((T + 1, top), -7, dtype=torch.int32, device=DEV)
    wt = torch.full((T + 1, top), -7.0, device=DEV)
    ops.moe_route(parts.to(DEV), groups, keep, top, 1.5, True, idx[:T], wt[:T], "chosen_softmax")
    best = logits.view(T, groups, -1).max(-1).values.sort(dim=-1, descending=True, stable=True).indices[:, :keep]
    kept = torch.zeros((T, groups), dtype=torch.bool).scatter_(1, best, True).repeat_interleave(E // groups, dim=1)
    able = min(top, keep * (E // groups))
    want = torch.where(kept, logits, -torch.inf).sort(dim=-1, descending=True, stable=True).indices[:, :able]
    assert torch.equal(idx[:T, :able].cpu().long(), want)
    assert (idx[:T, able:] == 0).all() and (wt[:T, able:] == 0).all()   # fewer eligible experts than choices: weight zero
    w = torch.exp(logits.gather(1, want).double())
    w = 1.5 * w / w.sum(-1, keepdim=True)
    # expf and each of the top additions err by two units of 2^-24 at most, the quotient and the scale by one each
    assert ((wt[:T, :able].cpu().double() - w).abs() <= (top + 8) * 2.0**-24 * w + 1e-12).all()
    assert (idx[T] == -7).all() and (wt[T] == -7).all()
