"""Which form a product takes at and around the number of tokens from which CTA pairs are taken always (no GPU)."""
from __future__ import annotations

from types import SimpleNamespace

import pytest

from inference_bench_b200.config.runtime_options import RuntimeOptions
from inference_bench_b200.kernels import gemm_tcgen05 as G

RT = SimpleNamespace(options=RuntimeOptions(), sm_count=148)


@pytest.mark.parametrize("T,n,k,add,form", [
    (2048, 4096, 4096, False, "pair"), (2048, 4096, 4096, True, "add"),     # 128 tiles: a tile a pair and more
    (2048, 64, 2048, False, "single"), (8192, 64, 2048, False, "single"),   # a router's scores
    (2048, 1024, 2048, True, "add"),                                        # added to the stream: always on pairs from here on
    (2304, 2048, 2816, False, "pair"), (2048, 2048, 2816, False, "pair"),   # few tiles, and the model keeps them on pairs
    (128, 64, 2048, False, "single"), (1, 4096, 4096, True, "single")])
def test_form(T, n, k, add, form):
    how = G.product_form(RT, T, n, k, add=add)
    assert how[0] == form
    if form == "single":   # a form that the kernel has, with no empty part of the k-range
        _, bn, splits, wide = how
        per = -(-(-(-k // 64)) // splits)
        assert bn in G.TOKEN_TILES and (splits - 1) * per < -(-k // 64) and (not wide or bn >= 128)


def test_one_sum_where_it_is_asked_for():
    """A head's product is never cut."""
    for T in (1, 64, 129, 2048, 4096):
        how = G.product_form(RT, T, 64, 2048, allow_split=False)
        assert how[0] == "pair" or how[2] == 1
