"""The choice of a token over vocabularies at the edges of a CTA's share and of the 16-byte accesses, with one to eight CTAs a row, and rows whose
thresholds fall on ties, on masked values or on nothing."""
from __future__ import annotations

import pytest
import torch

import plain_qwen3 as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CHOICES = [dict(), dict(temperature=0.7), dict(temperature=1.5, top_k=5), dict(temperature=1.0, top_p=0.6), dict(temperature=1.0, min_p=0.1),
           dict(temperature=0.8, top_k=20, top_p=0.95), dict(temperature=2.0, top_k=50, top_p=0.9, min_p=0.01), dict(temperature=1.0, top_p=1e-6), dict(temperature=1.0, top_p=0.999999)]


@pytest.mark.parametrize("V,rows", [(1, 9), (3, 9), (33, 9), (4095, 9), (4096, 9), (4097, 9), (8195, 18), (16388, 9), (32769, 9), (32768, 45), (40001, 9), (40000, 90), (9000, 160)])
def test_vocabularies(V, rows):
    from inference_bench_b200.kernels import ops
    from inference_bench_b200.sampling.params import SamplingParams
    g = torch.Generator().manual_seed(V + rows)
    logits = torch.randn(rows, V, generator=g) * 3
    params = [SamplingParams(seed=i, **CHOICES[i % len(CHOICES)]) for i in range(rows)]
    rows_dev = torch.tensor([p.row(i) for i, p in enumerate(params)], dtype=torch.int32, device=DEV)
    toks = torch.full((rows + 1,), -5, dtype=torch.int32, device=DEV)
    status = torch.tensor([7], dtype=torch.int32, device=DEV)
    ops.sample_rows(logits.to(DEV), rows_dev, toks, status)
    toks = toks.cpu().tolist()
    assert toks[rows] == 7
    few = range(rows) if V * rows < 400_000 else range(rows - 9, rows)   # the oracle is slow
    assert [toks[i] for i in few] == [P.sample_token(logits[i], p.temperature, p.seed, i, p.top_k, p.top_p, p.min_p) for i, p in enumerate(params) if i in few]


@pytest.mark.parametrize("V", [64, 20003])
def test_ties_and_masked_values(V):
    from inference_bench_b200.kernels import ops
    from inference_bench_b200.sampling.params import SamplingParams
    alike, masked, signed = torch.full((V,), 1.25), torch.full((V,), -torch.inf), torch.full((V,), -20.0)
    masked[V // 2], masked[V - 1] = 3.0, 3.0
    signed[V // 3], signed[V - 2] = 0.0, -0.0   # the best value twice, as zeros of both signs
    rows = [(logits, SamplingParams(seed=i, **choice)) for choice in CHOICES[1:] for i, logits in enumerate((alike, masked, signed))]
    params = torch.tensor([p.row(2) for _, p in rows], dtype=torch.int32, device=DEV)
    toks = torch.empty(len(rows), dtype=torch.int32, device=DEV)
    ops.sample_rows(torch.stack([x for x, _ in rows]).to(DEV), params, toks)
    assert toks.cpu().tolist() == [P.sample_token(x, p.temperature, p.seed, 2, p.top_k, p.top_p, p.min_p) for x, p in rows]


# rows at counts that give a row's cluster eight, four, two CTAs and one; vocabularies whose rows start on 16 bytes and ones whose rows do not
@pytest.mark.parametrize("V", [20000, 20003, 33001])
def test_a_row_does_not_depend_on_the_rows_beside_it(V):
    """Sharp cuts: unlike values of group A first, then many values alike, group B, which top-p takes in or leaves out by the last bits of A's mass."""
    from inference_bench_b200.kernels import ops
    from inference_bench_b200.sampling.params import SamplingParams
    g = torch.Generator().manual_seed(V)
    logits = torch.full((V,), -30.0)
    order = torch.randperm(V, generator=g)
    a, b = order[:V // 4], order[V // 4:V - 100]
    logits[a] = torch.rand(len(a), generator=g) * 2
    logits[b] = -0.5
    mass = torch.exp(logits.double() - logits.max().double())
    edge = float(mass[a].sum() / mass.sum())
    rows = [SamplingParams(temperature=1.0, seed=i, top_p=edge * (1 + k * 2.0**-24)).row(3) for i, k in enumerate(range(-20, 20))]
    alone = []
    for r in rows:
        t = torch.empty(1, dtype=torch.int32, device=DEV)
        ops.sample_rows(logits[None].to(DEV), torch.tensor([r], dtype=torch.int32, device=DEV), t)
        alone.append(t.item())
    in_b = torch.isin(torch.tensor(alone), b)
    assert in_b.any() and not in_b.all()   # the cut lies among these rows
    for count in (40, 80, 160):
        t = torch.empty(count, dtype=torch.int32, device=DEV)
        params = torch.tensor((rows * 4)[:count], dtype=torch.int32, device=DEV)
        ops.sample_rows(logits.expand(count, V).contiguous().to(DEV), params, t)
        assert t.tolist() == (alone * 4)[:count], f"{count} rows"
