"""The float32 path's product at the edges of their tiles."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import DEV, _g

pytestmark = pytest.mark.gpu


# tiles of 16 x 16, 16 x 64, 32 x 32, 32 x 64 and 64 x 64, with remainders in every size, inner sizes that no vector load takes, and the smallest
@pytest.mark.parametrize("T,N,K", [(1, 1, 1), (3, 17, 5), (16, 9473, 68), (15, 100, 200), (17, 16, 64), (100, 1531, 130), (129, 4799, 36), (333, 2050, 260), (640, 4100, 72), (70, 130, 41)])
@pytest.mark.parametrize("x_dtype,w_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16)])
def test_product_at_tile_edges(T, N, K, x_dtype, w_dtype):
    from inference_bench_b200.kernels import ops
    g = _g(T + N + K)
    x, w = torch.randn(T, K, generator=g).to(x_dtype).to(DEV), torch.randn(N, K, generator=g).to(w_dtype).to(DEV)
    out = torch.full((T, N), float("nan"), device=DEV)
    ops.gemm_simt(x, w, out)
    xd, wd = x.double(), w.double()
    # a chain of n FMAs is off by at most n eps times the sum of magnitudes; the longest of the four chains has ceil(K / 64) * 16 terms, two additions follow
    bound = (-(-K // 64) * 16 + 3) * 2.0 ** -24 * (xd.abs() @ wd.abs().T)
    assert ((out.double() - xd @ wd.T).abs() <= bound).all()
    # a row does not depend on how many others there are
    alone = torch.empty(1, N, device=DEV)
    ops.gemm_simt(x[-1:].contiguous(), w, alone)
    assert torch.equal(alone[0], out[-1])
