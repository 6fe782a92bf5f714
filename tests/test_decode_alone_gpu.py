"""Captured decode steps that fetch their inputs and leave their tokens themselves (`GpuExecutor.execute`) against those with copies around them."""
from __future__ import annotations

import pytest
import torch

from test_dense_layers_gpu import _runner

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [4, 1024, 1028, 40000])
def test_inputs_from_pinned_memory(n):
    from inference_bench_b200.kernels import lib as L, ops
    host = torch.arange(n, dtype=torch.int32).pin_memory()
    dev = torch.full((n + 4,), -1, dtype=torch.int32, device=DEV)
    for add in (0, 7):   # (what the host writes between two calls arrives)
        host.add_(add)
        ops.fetch_ints(host, dev[:n])
        assert torch.equal(dev[:n].cpu(), host) and (dev[n:] == -1).all()
    for bad in (host[:n - 1], torch.arange(n, dtype=torch.int32), host.long()):
        with pytest.raises(L.KernelError):
            ops.fetch_ints(bad, dev[:bad.shape[0]])


@pytest.mark.parametrize("batch", [1, 3, 8])
def test_the_same_tokens_with_and_without_copies(batch):
    """A few steps of a batch (padded to four rows where it has three), greedy and drawn: tokens, logits and cache."""
    from inference_bench_b200.engine.executor import GpuExecutor
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.sampling.params import GREEDY, SamplingParams
    got = []
    for alone in (True, False):
        r = _runner(256, 640, 4, 2, 64, 0, 16)
        ex, tokens = GpuExecutor(r), []
        for i in range(batch):
            r.cache.admit(i)
            r.step([StepEntry(i, list(range(3 + 5 * i)), [])])
        last = [7 + i for i in range(batch)]
        for step in range(5):
            entries = [StepEntry(i, [t], [0]) for i, t in enumerate(last)]
            sampling = [(GREEDY if i % 2 == 0 else SamplingParams(temperature=0.9, seed=i), step) for i in range(batch)]
            if alone:
                last = ex.execute(entries, sampling)
                logits = ex.last_logits
            else:
                handle = ex.launch_decode(entries, sampling)
                last = ex.collect(handle)
                logits = handle[0].logits
            tokens.append(last)
            tokens.append(logits[:batch].cpu())
        group = r.cache.groups[0]   # (the requests' own pages; the scratch page holds what padded rows left)
        pages = sorted({int(p) for i in range(batch) for p in r.cache.table(0, i) if p >= 0})
        got.append((tokens, group.tensor[:, pages].clone()))
        r.rt.check_status()
    for a, b in zip(got[0][0], got[1][0]):
        assert a == b if isinstance(a, list) else torch.equal(a, b)
    used = max(3 + 5 * i for i in range(batch)) + 5
    assert got[0][1].shape == got[1][1].shape and used <= 16 * got[0][1].shape[1] and torch.equal(got[0][1], got[1][1])


def test_a_bad_token_is_reported():
    """The status word comes back beside the tokens."""
    from inference_bench_b200.engine.executor import GpuExecutor
    from inference_bench_b200.engine.runtime import DeviceStatusError
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.kernels import lib as L
    from inference_bench_b200.sampling.params import GREEDY
    r = _runner(256, 640, 4, 2, 64, 0, 16)
    ex = GpuExecutor(r)
    r.cache.admit(0)
    ex.execute([StepEntry(0, [1], [0])], [(GREEDY, 0)])
    r.rt.status.fill_(L.ERR_BAD_TOKEN)
    with pytest.raises(DeviceStatusError):
        ex.execute([StepEntry(0, [1], [0])], [(GREEDY, 1)])
    assert isinstance(ex.execute([StepEntry(0, [1], [0])], [(GREEDY, 2)])[0], int)


@pytest.mark.parametrize("batch", [1, 3])
def test_tokens_left_by_one_form_feed_the_other(batch):
    """Steps that feed on the tokens left on the device, each behind a step that the host waited for, give the tokens that waiting for every step gives."""
    from inference_bench_b200.engine.executor import GpuExecutor
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.sampling.params import SamplingParams
    got = []
    for mixed in (False, True):
        r = _runner(256, 640, 4, 2, 64, 0, 16)
        ex, tokens = GpuExecutor(r), []
        for i in range(batch):
            r.cache.admit(i)
            r.step([StepEntry(i, list(range(5 + 7 * i)), [])])
        last = [9 + i for i in range(batch)]
        for step in range(6):
            sampling = [(SamplingParams(temperature=1.5, seed=3 + i), step) for i in range(batch)]
            if mixed and step % 2:
                last = ex.collect(ex.launch_decode([StepEntry(i, [0], [0]) for i in range(batch)], sampling, feed=True))
            else:
                last = ex.execute([StepEntry(i, [t], [0]) for i, t in enumerate(last)], sampling)
            tokens.append(last)
        got.append(tokens)
    assert got[0] == got[1]
    assert len(set(sum(got[0], []))) > 1
    g = ex.graph_for(batch)   # two captured forms over one set of buffers and one pool
    assert set(g.graphs) == {True, False} and len({x.pool() for x in g.graphs.values()}) == 1


def test_a_capture_outlives_a_garbage_collection():
    """Another graph becomes garbage in a cycle while a step is captured, and enough objects are made for the collector to run."""
    import gc
    from inference_bench_b200.engine.executor import GpuExecutor
    from inference_bench_b200.engine.step import StepEntry
    from inference_bench_b200.sampling.params import GREEDY
    x = torch.zeros(8, device=DEV)
    other = torch.cuda.CUDAGraph()
    with torch.cuda.graph(other):
        x.add_(1)
    held = [other]
    held.append(held)
    del other
    r = _runner(256, 640, 4, 2, 64, 0, 16)
    ex, forward = GpuExecutor(r), r.decoder.forward

    def dropping(ctx):
        nonlocal held
        if torch.cuda.is_current_stream_capturing():
            held = None
            made = [[] for _ in range(5000)]
            assert not gc.isenabled() and len(made) == 5000
        return forward(ctx)
    r.decoder.forward = dropping
    r.cache.admit(0)
    first = ex.execute([StepEntry(0, [1], [0])], [(GREEDY, 0)])
    assert held is None and gc.isenabled()
    assert ex.execute([StepEntry(0, first, [0])], [(GREEDY, 1)])
