"""Runs the scheduler's steps on the device: the step function, then sampling, tokens back to the host.

Steps that hold only decoded tokens are the launch-bound inner loop of generation, so they are
replayed as CUDA graphs, one per padded batch size (1, 2, 4, ... rows), like the reference's
`Stepper` (crates/specrt/src/runtime/step.rs:8-20, 197-228): all inputs of such a step live in one
static device buffer that a single copy (or the step itself) fills, padded rows write to a scratch page and a scratch
slot, and the graph holds the whole model, the sampling kernel included.
"""
from __future__ import annotations

import contextlib
import gc
from typing import Optional

import numpy as np
import torch

from ..kernels import ops
from ..sampling.params import SamplingParams
from ..sampling.sampler import Sampler
from .context import Segment, StepContext
from .step import ModelRunner, StepEntry


RUN_AHEAD_MAX = 64


@contextlib.contextmanager
def _no_collection():
    """A capture is lost when the garbage collector destroys another graph meanwhile (of an engine that is no longer used, say): the driver allows no such call
    while a stream is capturing. What is garbage now is collected afterwards."""
    on = gc.isenabled()
    gc.disable()
    try:
        yield
    finally:
        if on:
            gc.enable()


class _DecodeGraph:
    """The captured decode step for `rows` rows and the static buffers it reads and writes. It has two forms, each captured when it is first needed, over the
    same buffers and memory pool, so that a step of either form finds what the step before left on the device. alone: a step that the host waits for
    (`run`); it fetches its inputs from the pinned block and leaves its tokens there itself. Otherwise the inputs are copied in front of it (`launch`,
    `run_ahead`)."""

    def __init__(self, runner: ModelRunner, rows: int):
        self.runner, self.rows = runner, rows
        cache, rt = runner.cache, runner.rt
        B, W = rows, cache.table_width
        n_groups = len(cache.groups)
        # layout of the int32 input block: tokens | positions | seg_pos0 | seg_slot | params[B,6] | tables[g][B,W] | count
        self.n_ints = (4 * B + 6 * B + n_groups * B * W + 1 + 3) // 4 * 4
        self.host = torch.zeros(self.n_ints, dtype=torch.int32).pin_memory()
        self.dev = torch.zeros(self.n_ints, dtype=torch.int32, device=rt.device)
        h = self.host.numpy()
        self.h_tokens, self.h_pos, self.h_pos0, self.h_slot = h[0:B], h[B:2 * B], h[2 * B:3 * B], h[3 * B:4 * B]
        self.h_params = h[4 * B:10 * B].reshape(B, 6)
        self.h_tables = [h[10 * B + g * B * W:10 * B + (g + 1) * B * W].reshape(B, W) for g in range(n_groups)]
        d = self.dev
        self.d_tables = [d[10 * B + g * B * W:10 * B + (g + 1) * B * W].view(B, W) for g in range(n_groups)]
        const = torch.arange(B + 1, dtype=torch.int32, device=rt.device)
        segs = [Segment(None, cache.scratch_slot, 0, [0], [0]) for _ in range(B)]
        ar = np.arange(B, dtype=np.int32)
        self.ctx = StepContext(
            rt, segs, B, self.h_tokens, self.h_pos, ar, np.arange(B + 1, dtype=np.int32), self.h_pos0, self.h_slot, ar,
            token_ids=d[0:B], positions=d[B:2 * B], seg_of_token=const[:B], seg_start=const, seg_pos0=d[2 * B:3 * B], seg_slot=d[3 * B:4 * B],
            logit_rows=const[:B], caches=cache.views(self.d_tables))
        self.ctx.fixed_shape = True
        self.d_params = d[4 * B:10 * B].view(B, 6)
        self.d_count = d[self.n_ints - 1:self.n_ints]
        self.history = torch.zeros((RUN_AHEAD_MAX, B), dtype=torch.int32, device=rt.device)
        self.h_history = torch.zeros((RUN_AHEAD_MAX, B), dtype=torch.int32).pin_memory()
        self.result = torch.zeros(B + 1, dtype=torch.int32, device=rt.device)   # the step's tokens, then the status word after the step
        self.tokens = self.result[:B]
        self.h_out = torch.zeros(B + 1, dtype=torch.int32).pin_memory()
        self.np_out = self.h_out.numpy()
        # for steps launched without waiting (two may be in flight): a staging copy of the inputs, a place for the tokens and an event each (`capture`)
        self.stages: list[torch.Tensor] = []
        self.h_outs: list[torch.Tensor] = []
        self.events: list[torch.cuda.Event] = []
        self.pending = [False, False]
        self.turn = 0
        self.logits: Optional[torch.Tensor] = None   # of the step replayed last
        # by form: the captured step, its logits, the kernels in one replay
        self.graphs: dict[bool, torch.cuda.CUDAGraph] = {}
        self.logits_of: dict[bool, torch.Tensor] = {}
        self.launches: dict[bool, int] = {}
        self._pad_all()

    def _pad_all(self) -> None:
        cache = self.runner.cache
        self.h_tokens[:] = 0
        self.h_pos[:] = 0
        self.h_pos0[:] = 0
        self.h_slot[:] = cache.scratch_slot
        self.h_params[:] = 0
        for g, t in enumerate(self.h_tables):
            t[:] = cache.scratch_page(g)

    def _forward(self, alone: bool) -> torch.Tensor:
        self.ctx.memo = {}
        logits = self.runner.decoder.forward(self.ctx)
        ops.sample_rows(logits, self.d_params, self.result, self.runner.rt.status)
        c = self.ctx
        ops.advance_rows(self.tokens, c.token_ids, c.positions, c.seg_pos0, self.d_params, self.history, self.d_count, self.h_out if alone else None)
        return logits

    def capture(self, alone: bool) -> None:
        """Capture one form. The second form runs nothing on the device (a step of the first may have left tokens there) and takes its memory from the first's
        pool: a replay's intermediates are dead when it ends, and replays follow one another on one stream."""
        self.runner.rt.activate()
        if not self.graphs:
            ops.fetch_ints(self.host, self.dev)
            stream = torch.cuda.Stream(device=self.runner.rt.device)
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                for _ in range(2):   # warm-up outside the capture: lazy kernel attributes, allocator
                    self._forward(alone)
            torch.cuda.current_stream().wait_stream(stream)
        if not alone and not self.stages:
            self.stages = [torch.zeros(self.n_ints, dtype=torch.int32).pin_memory() for _ in range(2)]
            self.h_outs = [torch.zeros(self.rows + 1, dtype=torch.int32).pin_memory() for _ in range(2)]
            self.events = [torch.cuda.Event() for _ in range(2)]
        torch.cuda.synchronize()
        from ..kernels import lib
        before = lib.launches
        graph = torch.cuda.CUDAGraph()
        with _no_collection(), torch.cuda.graph(graph, pool=next(iter(self.graphs.values())).pool() if self.graphs else None):
            if alone:
                ops.fetch_ints(self.host, self.dev)
            self.logits_of[alone] = self._forward(alone)
        self.graphs[alone] = graph
        self.launches[alone] = lib.launches - before

    def _replay(self, alone: bool) -> None:
        self.graphs[alone].replay()
        self.logits = self.logits_of[alone]

    def run_ahead(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]], steps: int) -> list[list[int]]:
        """`steps` decode steps with no host work in between: every step's sampled tokens are the next
        step's inputs on the device. The requests' pages for all `steps` positions must be allocated.
        Returns the tokens of every step, [steps][rows]."""
        if not 1 <= steps <= RUN_AHEAD_MAX:
            raise ValueError(f"run_ahead takes 1 to {RUN_AHEAD_MAX} steps, got {steps}")
        reqs = [e.request for e in entries]
        self._fill(entries, sampling, reqs, self.runner.cache.rows(reqs))
        self.dev.copy_(self.host, non_blocking=True)
        for _ in range(steps):
            self._replay(False)
        self.h_history.copy_(self.history, non_blocking=True)
        self.h_out.copy_(self.result, non_blocking=True)
        torch.cuda.current_stream(self.runner.rt.device).synchronize()
        self.runner.rt.raise_for(int(self.h_out[self.rows]))
        return self.h_history[:steps, :len(entries)].tolist()

    def run(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]], reqs: list, rows) -> list[int]:
        """reqs, rows: the entries' requests and their slots (`CacheManager.rows`)."""
        self._fill(entries, sampling, reqs, rows)
        self._replay(True)
        torch.cuda.current_stream(self.runner.rt.device).synchronize()
        out = self.np_out.tolist()
        self.runner.rt.raise_for(out[self.rows])
        return out[:len(entries)]

    def launch(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]], feed: bool, reqs: list, rows) -> tuple[int, int]:
        """Enqueue one step and return at once. With `feed` the input tokens stay what the step before
        left on the device (its sampled tokens, row by row): everything but the tokens is copied."""
        slot = self.turn
        if self.pending[slot]:
            raise RuntimeError("two decode steps are already in flight")
        self.turn ^= 1
        self._fill(entries, sampling, reqs, rows, tokens=not feed)
        stage = self.stages[slot]
        stage.copy_(self.host)
        if feed:
            self.dev[self.rows:].copy_(stage[self.rows:], non_blocking=True)
        else:
            self.dev.copy_(stage, non_blocking=True)
        self._replay(False)
        self.h_outs[slot].copy_(self.result, non_blocking=True)
        self.events[slot].record()
        self.pending[slot] = True
        return slot, len(entries)

    def collect(self, handle: tuple[int, int]) -> list[int]:
        slot, n = handle
        self.events[slot].synchronize()
        self.pending[slot] = False
        self.runner.rt.raise_for(int(self.h_outs[slot][self.rows]))
        return self.h_outs[slot][:n].tolist()

    def _fill(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]], reqs: list, rows, tokens: bool = True) -> None:
        cache = self.runner.cache
        n = len(entries)
        if n < self.rows:
            self._pad_all()
        slots = cache.fill_rows(reqs, self.h_pos, self.h_tables, rows)   # positions and block tables, straight into the pinned block
        if tokens:
            self.h_tokens[:n] = [e.tokens[0] for e in entries]
        self.h_pos0[:n] = self.h_pos[:n]
        self.h_slot[:n] = slots
        params, last = [], (None, None, None)
        for p, step in sampling:   # (requests that were started together share a row)
            if p is not last[0] or step != last[1]:
                last = (p, step, p.row(step))
            params.append(last[2])
        self.h_params[:n] = params


class GpuExecutor:
    def __init__(self, runner: ModelRunner, use_graphs: bool = True, max_graph_rows: int = 256):
        self.runner = runner
        self.sampler = Sampler(runner.rt.device)
        self.use_graphs, self.max_graph_rows = use_graphs, max_graph_rows
        self._graphs: dict[int, _DecodeGraph] = {}
        self.last_logits: Optional[torch.Tensor] = None
        self.steps = 0
        self.h2d_bytes = 0
        self.d2h_bytes = 0

    def graph_for(self, n_rows: int, alone: bool = True) -> _DecodeGraph:
        """The captured step for this many rows, with the form of `execute` or that of `launch_decode` and `decode_ahead` captured."""
        rows = 1
        while rows < n_rows:
            rows *= 2
        g = self._graphs.get(rows)
        if g is None:
            g = self._graphs[rows] = _DecodeGraph(self.runner, rows)
        if alone not in g.graphs:
            g.capture(alone)
        return g

    def decode_ahead(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]], steps: int) -> list[list[int]]:
        """Several decode steps of the same requests in a row, tokens fed back on the device."""
        cache = self.runner.cache
        g = self.graph_for(len(entries), alone=False)
        reqs = [e.request for e in entries]
        rows = cache.rows(reqs)
        cache.extend_rows(reqs, rows, steps)
        out = g.run_ahead(entries, sampling, steps)
        cache.commit_rows(reqs, rows, steps)
        self.steps += steps
        self.h2d_bytes += g.n_ints * 4
        self.d2h_bytes += steps * g.rows * 4 + 4
        return out

    def launch_decode(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]], feed: bool = False):
        """Enqueue a step of single decoded tokens without waiting for it; `collect` returns its tokens.
        With `feed`, every row's input token is the one the step before sampled for it, taken on the
        device. None when such a step cannot run as a graph. Raises OutOfPages with nothing changed."""
        if not self.use_graphs or len(entries) > self.max_graph_rows:
            return None
        cache = self.runner.cache
        if not feed:
            for e in entries:
                if not 0 <= e.tokens[0] < self.runner.vocab:
                    raise ValueError(f"request {e.request!r}: token id {e.tokens[0]} is outside the vocabulary of {self.runner.vocab}")
        g = self.graph_for(len(entries), alone=False)
        reqs = [e.request for e in entries]
        rows = cache.rows(reqs)
        try:
            cache.extend_rows(reqs, rows, 1)
        except Exception:
            for req in reqs:
                cache.shrink_to_committed(req)
            raise
        handle = g.launch(entries, sampling, feed, reqs, rows)
        cache.commit_rows(reqs, rows, 1)
        self.steps += 1
        self.h2d_bytes += (g.n_ints - (g.rows if feed else 0)) * 4
        self.d2h_bytes += g.rows * 4 + 4
        return g, handle

    def collect(self, handle) -> list[int]:
        g, h = handle
        return g.collect(h)

    def execute(self, entries: list[StepEntry], sampling: list[tuple[SamplingParams, int]]) -> list[int]:
        self.steps += 1
        cache = self.runner.cache
        if self.use_graphs and len(entries) <= self.max_graph_rows and all(len(e.tokens) == 1 and len(e.want) == 1 and e.want[0] == 0 for e in entries):
            g = self.graph_for(len(entries))
            vocab = self.runner.vocab
            for e in entries:
                if not 0 <= e.tokens[0] < vocab:
                    raise ValueError(f"request {e.request!r}: token id {e.tokens[0]} is outside the vocabulary of {vocab}")
            reqs = [e.request for e in entries]
            rows = cache.rows(reqs)     # a step's bookkeeping is one call into the core each, not one a request
            cache.extend_rows(reqs, rows, 1)
            out = g.run(entries, sampling, reqs, rows)
            cache.commit_rows(reqs, rows, 1)
            self.last_logits = g.logits
            self.h2d_bytes += g.n_ints * 4
            self.d2h_bytes += g.rows * 4 + 4
            return out
        logits = self.runner.step(entries, check=False)
        if logits is None:   # nothing to sample: no transfer comes back, so the status word is read when a later step's tokens are
            return []
        tokens = self.sampler.sample(logits, [p for p, _ in sampling], [s for _, s in sampling], self.runner.rt.status)
        self.last_logits = logits
        self.h2d_bytes += sum(len(e.tokens) for e in entries) * 12 + len(entries) * (12 + 4 * cache.table_width * len(cache.groups)) + len(sampling) * 28
        self.d2h_bytes += len(sampling) * 4 + 4
        host = tokens.cpu().tolist()
        self.runner.rt.raise_for(host[-1])
        return host[:-1]
