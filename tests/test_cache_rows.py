"""The cache manager's calls for all rows of a step against the calls for one request."""
import random

import numpy as np
import pytest

from inference_bench_b200.cache.manager import CacheError, CacheManager, OutOfPages
from inference_bench_b200.parts.base import FixedState, PagedKV


def _manager(pages=12):
    return CacheManager([PagedKV(2, 8, None), PagedKV(2, 8, 6), FixedState((5,))], 4, pages, 4, 40)


def _state(m):
    return [m.length(r) for r in m.live()], [t.tolist() for t in m._tables], m.used_pages()


@pytest.mark.parametrize("seed", range(5))
def test_rows_do_what_single_calls_do(seed):
    rng = random.Random(seed)
    a, b = _manager(), _manager()
    for step in range(60):
        if a.free_slots() and rng.random() < 0.4:
            a.admit(step), b.admit(step)
        reqs = [r for r in a.live() if rng.random() < 0.7]
        by = rng.choice([1, 1, 1, 3, 9])
        errors = []
        try:
            for r in reqs:
                a.extend(r, a.length(r) + by)
        except OutOfPages as e:
            errors.append(str(e))
        rows = b.rows(reqs)
        try:
            b.extend_rows(reqs, rows, by)
        except OutOfPages as e:
            errors.append(str(e))
        assert len(errors) in (0, 2) and len(set(errors)) <= 1 and _state(a) == _state(b)      # the same refusal at the same request
        if errors:
            for r in reqs:
                a.shrink_to_committed(r), b.shrink_to_committed(r)
        else:
            for r in reqs:
                a.commit(r, a.length(r) + by)
            b.commit_rows(reqs, rows, by)
            pos = np.zeros(4, np.int32)
            tables = [np.full((4, b.table_width), -7, np.int32) for _ in b.groups]
            assert b.fill_rows(reqs, pos, tables, rows) == [a.slot(r) for r in reqs] == b.fill_rows(reqs, pos, tables)
            assert pos[:len(reqs)].tolist() == [a.length(r) for r in reqs]
        assert _state(a) == _state(b)
        if a.live() and rng.random() < 0.3:
            r = rng.choice(a.live())
            a.release(r), b.release(r)
        a.check(), b.check()


def test_unknown_requests_are_refused():
    m = _manager()
    m.admit("a")
    with pytest.raises(CacheError, match="'b' is not admitted"):
        m.rows(["a", "b"])
    rows = m.rows(["a"])
    m.release("a")
    with pytest.raises(CacheError):
        m.commit_rows(["a"], rows, 1)
    with pytest.raises(CacheError):
        m.extend_rows(["a"], rows, 1)
