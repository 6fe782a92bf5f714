"""What one step looks like to the parts: the tokens of the batch and where each one lives.

A batch is a list of segments; a segment is a run of consecutive tokens of one request, starting
at position `pos0` (a decoded token is a segment of length 1). All tokens of all segments form one
flat batch of T rows. The reference's row records are `DecodeRow{slot, token, pos}` and
`PrefillPart{slot, tokens, start}` (crates/specrt/src/runtime/step.rs:23-29,
crates/specrt/src/runtime/fused.rs:6-11); here any number of either may share a step.
"""
from __future__ import annotations

from dataclasses import dataclass, field
from functools import cached_property
from typing import Any, Optional, Sequence

import numpy as np
import torch

from ..kernels import attention
from .runtime import Runtime


@dataclass
class Segment:
    request: Any          # the request's id
    slot: int             # its state slot
    pos0: int             # position of its first token in this step
    tokens: Sequence[int]
    want: Sequence[int] = ()   # places among `tokens` whose logits are wanted


@dataclass
class StepContext:
    rt: Runtime
    segments: list[Segment]
    n_tokens: int
    # host copies (numpy int32)
    h_token_ids: np.ndarray
    h_positions: np.ndarray
    h_seg_of_token: np.ndarray
    h_seg_start: np.ndarray      # [S+1] offsets into the flat batch
    h_seg_pos0: np.ndarray       # [S]
    h_seg_slot: np.ndarray       # [S]
    h_logit_rows: np.ndarray     # [K] flat row index of every wanted place, in entry order
    # device copies (int32)
    token_ids: torch.Tensor
    positions: torch.Tensor
    seg_of_token: torch.Tensor
    seg_start: torch.Tensor
    seg_pos0: torch.Tensor
    seg_slot: torch.Tensor
    logit_rows: torch.Tensor
    # per schedule entry: what the cache manager gives that execution (KvLayerView, StateView or None)
    caches: list = field(default_factory=list)
    # parts may keep per-step results here (e.g. rotation tables shared by all layers)
    memo: dict = field(default_factory=dict)
    # the step's block tables on the device, where `build_context` was given them
    tables: list = field(default_factory=list)
    # True when the step is being captured into (or replayed from) a CUDA graph: launch shapes must
    # then depend on the batch's sizes only, never on the host copies of positions or tables
    fixed_shape: bool = False
    # None, or a list that the decoder fills with the residual stream at the wanted rows: after the embedding, then after
    # every schedule entry (float32 [wanted, hidden] each). Debugging only.
    trace: Optional[list] = None

    @property
    def n_segments(self) -> int:
        return len(self.segments)

    @cached_property   # (asked several times a layer)
    def max_segment_len(self) -> int:
        return int((self.h_seg_start[1:] - self.h_seg_start[:-1]).max()) if self.segments else 0


def build_context(rt: Runtime, segments: list[Segment], caches: Optional[list] = None, tables: Optional[list] = None) -> StepContext:
    """Flatten segments into the arrays of a step and copy them to the device in one transfer. tables: the step's block tables (int32 [segments, width]
    each), for a caller that makes the caches' views from them (`StepContext.tables`): they and the attention kernels' work lists travel along."""
    S = len(segments)
    lens = [len(s.tokens) for s in segments]
    starts, T, rows = [0], 0, []
    for s, n in zip(segments, lens):
        for w in s.want:
            if not 0 <= w < n:
                raise ValueError(f"request {s.request!r}: wanted place {w} is outside its {n} tokens of this step")
            rows.append(T + int(w))
        T += n
        starts.append(T)
    dec, longest, tile_seg, tile_row0, tile_keys = attention.work_lists(lens, starts, [s.pos0 for s in segments]) if tables else ([], None, [], [], 0)
    # one pinned staging buffer, one copy; the host's arrays are the buffer's parts
    sizes = [T, T, T, S + 1, S, S, len(rows), len(dec), len(tile_seg), len(tile_seg)]
    total = sum(sizes)
    sizes.append(-total % 4)   # (tables start on 16 bytes)
    for t in tables or ():
        sizes += [t.size, -t.size % 4]
    staging = torch.empty(max(sum(sizes), 1), dtype=torch.int32, pin_memory=True)
    flat = staging.numpy()
    token_ids, positions, seg_of_token = flat[:T], flat[T:2 * T], flat[2 * T:3 * T]
    o = 3 * T
    seg_start, seg_pos0, seg_slot = flat[o:o + S + 1], flat[o + S + 1:o + 2 * S + 1], flat[o + 2 * S + 1:o + 3 * S + 1]
    o += 3 * S + 1
    logit_rows = flat[o:o + len(rows)]
    flat[o:total] = rows + dec + tile_seg + tile_row0
    seg_start[:], seg_pos0[:], seg_slot[:] = starts, [s.pos0 for s in segments], [s.slot for s in segments]
    for s, a, n in zip(segments, starts, lens):
        if n == 1:
            token_ids[a] = s.tokens[0]
        elif n:
            token_ids[a:a + n] = s.tokens
    if S == 1:
        seg_of_token[:] = 0
        positions[:] = np.arange(segments[0].pos0, segments[0].pos0 + T, dtype=np.int32)
    elif T:
        seg_of_token[:] = np.repeat(np.arange(S, dtype=np.int32), lens)
        np.add(np.repeat(seg_pos0 - seg_start[:-1], lens), np.arange(T, dtype=np.int32), out=positions)
    o = total + sizes[10]
    for t in tables or ():
        flat[o:o + t.size] = t.reshape(-1)
        o += t.size + -t.size % 4
    dev = staging.to(rt.device, non_blocking=True)
    views = dev[:sum(sizes)].split(sizes)
    ctx = StepContext(rt, segments, T, token_ids, positions, seg_of_token, seg_start, seg_pos0, seg_slot, logit_rows, *views[:7], caches=caches or [])
    if tables:
        ctx.tables = [views[11 + 2 * i].view(t.shape) for i, t in enumerate(tables)]
        ctx.memo[attention.WORK_KEY] = attention.device_work(views[7], views[8], views[9], longest, tile_keys)
    return ctx
