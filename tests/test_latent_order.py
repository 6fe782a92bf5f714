"""Where a launch without programmatic dependence stands in a step with prompt portions (no GPU)."""
from __future__ import annotations

import threading


def test_the_mark_for_the_next_launch_is_the_threads_own():
    """Another thread's launch in between does not use it up."""
    from inference_bench_b200.kernels import lib
    core, other = lib.load(), []
    core.ib_set_pdl(1)
    core.ib_pdl_skip_next()
    t = threading.Thread(target=lambda: other.append(core.ib_pdl_enabled()))
    t.start()
    t.join()
    assert other == [1] and core.ib_pdl_enabled() == 0 and core.ib_pdl_enabled() == 1
