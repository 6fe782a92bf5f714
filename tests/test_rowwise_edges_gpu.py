"""SiLU-mul and the embedding around the sizes at which their 16-byte forms begin and end (csrc/elementwise.cu)."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import DEV, _g, status  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


# inner sizes of one thread, around a CTA's 512 values, and one that four does not divide; partial sums around the four that are requested together
@pytest.mark.parametrize("T,I", [(1, 4), (3, 508), (65, 512), (2, 516), (5, 510), (1, 3072)])
@pytest.mark.parametrize("P", [1, 4, 5, 6])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_silu_mul(T, I, P, dtype):
    from inference_bench_b200.kernels import ops
    gu = torch.randn((P, T, 2 * I), generator=_g(T + I + P)).to(DEV)
    act = torch.full((T + 1, I), 7.0, device=DEV, dtype=dtype)
    ops.silu_mul(gu, act[:T])
    s = gu.double().sum(0)
    g, u = s[:, :I], s[:, I:]
    want = g * torch.sigmoid(g) * u
    # both sums are off by at most P 2^-24 of their terms' sizes, the exponential and division by a few 2^-23, one rounding to bfloat16
    size = gu.double().abs().sum(0)
    bound = (P + 4) * 2.0 ** -23 * (size[:, :I] * (1 + u.abs()) + size[:, I:] * g.abs()) + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs()
    assert ((act[:T].double() - want).abs() <= bound).all() and (act[T:] == 7.0).all()


# from 2^18 partial sums on a thread has four neighbours: inner sizes that end inside a CTA's 512, at it and behind it; partial sums around the five that are
# requested together and the four behind them
@pytest.mark.parametrize("T,I", [(2100, 132), (520, 508), (512, 512), (300, 1028), (90, 3072), (700, 510)])
@pytest.mark.parametrize("P", [1, 2, 5, 6, 10])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_silu_mul_of_many(T, I, P, dtype):
    test_silu_mul(T, I, P, dtype)


@pytest.mark.parametrize("H", [8, 504, 520, 4096, 4104, 12, 7])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embed(status, H, dtype):  # noqa: F811
    from inference_bench_b200.kernels import ops
    table = torch.randn((33, H), generator=_g(H)).to(dtype).to(DEV)
    tokens = torch.tensor([32, 0, 5, 5, 17], dtype=torch.int32, device=DEV)
    x = torch.full((6, H), 7.0, device=DEV)
    ops.embed(table, tokens, x[:5], status)
    assert torch.equal(x[:5], table[tokens.long()].float()) and (x[5:] == 7.0).all() and status.item() == 0
    ops.embed(table, torch.tensor([33], dtype=torch.int32, device=DEV), x[:1], status)
    assert status.item() != 0
    status.zero_()
