"""The step function: one batch of (request, its next tokens) through the model, from the cache.

A step takes portions of prompts beside single decoded tokens, cut anywhere, runs exactly the
tokens it is given as one flat batch and returns the logits at the wanted places. The reference has
three entry points for this (prefill_slot, decode, fused_step: crates/specrt/src/runtime/step.rs:121-232,
crates/specrt/src/runtime/fused.rs:14-61) and allows one prompt portion beside decode rows; here one
function takes any mix.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Any, Hashable, Optional, Sequence

import numpy as np
import torch

from ..cache.manager import CacheManager
from ..parts.decoder import Decoder
from .context import Segment, StepContext, build_context
from .runtime import Runtime


@dataclass
class StepEntry:
    request: Hashable
    tokens: Sequence[int]
    want: Sequence[int] = ()


class ModelRunner:
    """Owns nothing but the wiring: a bound decoder, a cache manager and a runtime."""

    def __init__(self, decoder: Decoder, cache: CacheManager, rt: Runtime):
        self.decoder, self.cache, self.rt = decoder, cache, rt
        self.vocab = decoder.plan.vocab_size

    def step(self, entries: Sequence[StepEntry], check: bool = True, trace: Optional[list] = None) -> Optional[torch.Tensor]:
        """Run one step. Requests must be admitted to the cache manager; every entry continues its
        request where the last step left it. Returns float32 logits [wanted, vocab] on the device in
        the order of the entries and of their `want`, or None when nothing is wanted.
        Raises OutOfPages (and changes nothing) if a request cannot get its pages. `trace`: a list that receives the
        residual stream at the wanted rows after the embedding and after every schedule entry (debugging)."""
        entries = [e for e in entries if len(e.tokens) > 0]
        if not entries:
            return None
        self.rt.activate()
        reqs, tokens, vocab = [e.request for e in entries], [], self.vocab
        if len(set(reqs)) != len(reqs):
            twice = next(r for i, r in enumerate(reqs) if r in reqs[:i])
            raise ValueError(f"request {twice!r} appears twice in one step")
        for e in entries:
            if len(e.tokens) == 1:
                toks = e.tokens
                lo = hi = toks[0]
            else:
                toks = np.asarray(e.tokens)
                lo, hi = toks.min(), toks.max()
            if lo < 0 or hi >= vocab:
                toks = np.asarray(toks)
                raise ValueError(f"request {e.request!r}: token id {int(toks[(toks < 0) | (toks >= vocab)][0])} is outside the vocabulary of {vocab}")
            tokens.append(toks)
        # pages first, all or nothing across the batch
        cache, lengths, done = self.cache, [self.cache.length(r) for r in reqs], []
        try:
            for r, toks, at in zip(reqs, tokens, lengths):
                cache.extend(r, at + len(toks))
                done.append(r)
        except Exception:
            for r in done:  # give back what this step took: shrink to the committed length
                cache.shrink_to_committed(r)
            raise
        segments = [Segment(e.request, cache.slot(e.request), at, toks, e.want) for e, toks, at in zip(entries, tokens, lengths)]
        ctx = build_context(self.rt, segments, tables=cache.step_tables(reqs))
        ctx.caches = cache.views(ctx.tables)
        ctx.trace = trace
        logits = self.decoder.forward(ctx)
        for r, toks, at in zip(reqs, tokens, lengths):
            cache.commit(r, at + len(toks))
        if check:
            self.rt.check_status()
        return logits
