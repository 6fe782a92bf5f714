"""Latent attention: keys and values of all heads are linear maps of one small latent per token, and only that latent
and one rotated key part shared by the heads are cached.

With h the layer's input, per token:
    q = Wq h, per head [q_n (dim) | q_r (rot_dim)];   [c_raw (kv_rank) | r_raw (rot_dim)] = Wdkv h;
    c = w_c * c_raw / rms(c_raw),  r = turn(r_raw),  q_r <- turn(q_r)      (pairs 2i, 2i+1; angle pos * base^(-2i/dims))
    head a:  k = Wuk_a c,  v = Wuv_a c,  s_j = (q_n . k_j + q_r . r_j) * scale  over j <= own position,  o_a = sum_j softmax(s)_j v_j
    out = Wo [o_1 | o_2 | ...]
The cache row of a token is [c | r]. The kernels never build k and v: q_n . (Wuk_a c) = (Wuk_a^T q_n) . c and
sum_j p_j Wuv_a c_j = Wuv_a (sum_j p_j c_j), so a head's query becomes [Wuk_a^T q_n | q_r] against the cached rows, and the
weighted sum of latents goes through Wuv_a afterwards (two small per-head products around one attention kernel that reads
kv_rank + rot_dim values a key for all heads together). That is the form for decoded tokens. A prompt portion has many queries a key: its
requests' k and v are made once a step (one product over the rows that the portion sees) and a kernel with the shape of grouped attention
reads them (csrc/latent_prefill.cu); which way a request's tokens go is decided by `_expanded`. A layer with own_kv=False has no Wdkv and reads the rows another
layer cached.

Variants, each a constructor parameter. `q_rank` n: the queries go through a latent of their own, c_q = w_q * rms_unit(Wdq h) (n values),
q = Wuq c_q; the layer's first product is then [Wdq | Wdkv] h and a second one makes the heads' queries. `window` W: a position sees
itself and the W - 1 positions before it (the cache then keeps only those pages). `gate`: head a's output is multiplied by
sigmoid(Wg h)_a, one number a head from the layer's input (its rows ride in the first product; the sigmoid sits in the epilogue of the
per-head product with Wuv). `sink`: a learned number per head whose exponential the softmax's denominator holds as well (no key, no value, not
scaled). rot_dim 0: no rotated part at all (the position encoding is then "none").
"""
from __future__ import annotations

from typing import Optional

import numpy as np
import torch

from ..kernels import ops
from . import base
from .base import PagedRows, WeightSpec


# A request's tokens of a step go through keys and values made per head from this many tokens on, while its context is at most so many times
# as long (making a key's heads costs as much as about a dozen of its pairs with a query), and while the step's rows keep the keys and
# values of one layer below this many bytes.
EXPAND_MIN_TOKENS, EXPAND_MAX_CONTEXT, EXPAND_MAX_BYTES = 32, 64, 1 << 29
# Where all other tokens of such a step may go the same way too, they do: one form costs less than two. Where some need the form that reads the
# latents (decoded tokens with long contexts), both forms run, three kernels more than the second alone: the portions must then save at least
# this many microseconds by the estimate of `_saved`. Whole passes of one layer beside 8 decoded tokens, the second form alone and both, us: heads
# of 64 + 32 on a latent of 256, 300 tokens 362 and 423, 1,000 426 and 446, 1,500 473 and 468, 2,048 531 and 488; 16 heads of 128 + 64 on 512,
# 300 tokens 385 and 422, 600 431 and 435, 1,000 507 and 458, 2,048 858 and 552.
EXPAND_BESIDE_SAVED_US = 60.0
# Multiplies a microsecond, from the kernels alone at portions of 512 to 2,048 tokens of both sizes: the maps to the latents' space and back, attention
# there, the product of keys and values, attention over them.
MAP_RATE, LATENT_RATE, MAKE_RATE, PAIR_RATE = 60e6, 53e6, 500e6, 400e6


def _runs(ranges, per: int) -> list:
    """The tokens a .. b - 1 of every range in runs of up to `per`: first, how many, first, how many ... in order."""
    out = []
    for a, b in ranges:
        whole = b - (b - a) % per
        for t in range(a, whole, per):
            out += (t, per)
        if whole < b:
            out += (whole, b - whole)
    return out


@base.register_mixer("latent_attention")
class LatentAttention(base.Mixer):
    def __init__(self, prefix: str, hidden: int, heads: int, dim: int, rot_dim: int, vdim: int, kv_rank: int, scale: float, norm_eps: float,
                 position: base.PositionEncoding, own_kv: bool = True, window: Optional[int] = None,
                 names: tuple = ("q", "dkv", "dkv.norm", "uk", "uv", "o", "dq", "dq.norm", "uq", "g", "sink"), q_rank: Optional[int] = None, gate: bool = False,
                 sink: bool = False):
        if getattr(position, "pairing", "interleaved") != "interleaved":
            raise ValueError("latent attention turns entry 2i with 2i + 1: it needs a position encoding with pairing=\"interleaved\" (or none)")
        if window is not None and (window <= 0 or not own_kv):
            raise ValueError("a window must be positive, and a layer that reads another layer's rows takes that layer's window")
        if q_rank is not None and (q_rank <= 0 or not own_kv):
            raise ValueError("a query latent must have a positive size, and is built for layers that keep their own latent")
        self.window, self.q_rank, self.gate = window, q_rank, bool(gate)
        self.w_uq = self.q_norm = None
        self.sink, self.sink_dev = bool(sink), None
        self.prefix, self.hidden, self.heads, self.dim, self.rot_dim, self.vdim, self.kv_rank = prefix, hidden, heads, dim, rot_dim, vdim, kv_rank
        self.scale, self.norm_eps, self.position, self.own_kv, self.names = scale, norm_eps, position, own_kv, tuple(names)
        self.w_kv = None      # [k rows of all heads | v rows of all heads] over the latent, where portions go through keys and values per head
        self.w_in = self.wuk_t = self.wuv = self.wo = self.c_norm = None

    def cache_need(self):
        return PagedRows(self.kv_rank + self.rot_dim, self.window) if self.own_kv else None

    def _name(self, i: int) -> str:
        return f"{self.prefix}.{self.names[i]}"

    def weight_specs(self):
        H, r = self.heads, self.kv_rank
        specs = [WeightSpec(self._name(3), (H * self.dim, r)), WeightSpec(self._name(4), (H * self.vdim, r)), WeightSpec(self._name(5), (self.hidden, H * self.vdim))]
        if self.q_rank is None:
            specs.append(WeightSpec(self._name(0), (H * (self.dim + self.rot_dim), self.hidden)))
        else:
            specs += [WeightSpec(self._name(6), (self.q_rank, self.hidden)), WeightSpec(self._name(7), (self.q_rank,), role="norm"),
                      WeightSpec(self._name(8), (H * (self.dim + self.rot_dim), self.q_rank))]
        if self.gate:
            specs.append(WeightSpec(self._name(9), (H, self.hidden)))
        if self.sink:
            specs.append(WeightSpec(self._name(10), (H,), std=1.0))
        if self.own_kv:
            specs += [WeightSpec(self._name(1), (r + self.rot_dim, self.hidden)), WeightSpec(self._name(2), (r,), role="norm")]
        return specs

    def bind(self, weights, rt):
        H, r = self.heads, self.kv_rank
        rows = [weights[self._name(0) if self.q_rank is None else self._name(6)]]
        if self.own_kv:
            rows.append(weights[self._name(1)])
            self.c_norm = rt.vector(weights[self._name(2)])
        if self.gate:
            rows.append(weights[self._name(9)])
        self.w_in = rt.matrix(torch.cat(rows, dim=0))   # [q of all heads (or the query latent) | latent | key part | gates] rows: one product for the layer's input
        if self.q_rank is not None:
            self.w_uq, self.q_norm = rt.matrix(weights[self._name(8)]), rt.vector(weights[self._name(7)])
        self.wuk_t = rt.upload(weights[self._name(3)].view(H, self.dim, r).transpose(1, 2), rt.act_dtype)   # [H, rank, dim]: q_n -> rank values
        self.wuv = rt.upload(weights[self._name(4)].view(H, self.vdim, r), rt.act_dtype)                    # [H, vdim, rank]
        if (rt.options.latent_attention == "auto" and rt.options.expert_gemm != "simt" and rt.act_dtype == torch.bfloat16 and rt.gemm != "simt" and self.scale > 0
                and self._tensor_cores(rt) and ops.latent_prefill_supports(self.dim, self.rot_dim, self.vdim, r)):
            self.w_kv = rt.upload(torch.cat([weights[self._name(3)], weights[self._name(4)]], dim=0), rt.act_dtype)
        self.wo = rt.matrix(weights[self._name(5)])
        if self.sink:
            self.sink_dev = rt.vector(weights[self._name(10)])
        self.position.bind(weights, rt)

    def _slices(self, ctx, view) -> tuple[int, int]:
        """(slices, keys per slice) of the attention kernel: a step of single decoded tokens has few (token, head block)
        pairs, so each one's keys are cut until every SM has two CTAs; a step with prompt portions has enough rows.
        The cut depends on the step's sizes (and, outside a captured step, its longest context) only."""
        key = ("latent slices", self.heads, self.window)
        if key not in ctx.memo:
            single = ctx.fixed_shape or ctx.max_segment_len == 1
            out = (1, 1 << 30)
            if single:
                max_keys = view.table_stride * view.page_size if ctx.fixed_shape else int(np.max(ctx.h_positions)) + 1
                if self.window is not None:
                    max_keys = min(max_keys, self.window)
                ctas = ctx.n_tokens * -(-self.heads // (16 if self._tensor_cores(ctx.rt) else 8))
                n = max(1, min(ctx.rt.sm_count // ctas, -(-max_keys // 128)))   # two key tiles a slice at least: the second arrives while the first is used
                if n > 1:
                    per = -(-(-(-max_keys // n)) // 64) * 64
                    out = (-(-max_keys // per), per)
            ctx.memo[key] = out
        return ctx.memo[key]

    def _rows_and_units(self, ctx):
        """For the tensor-core kernel: (query rows a CTA holds, runs of consecutive tokens of one request that fill them as int32 [n, 2]
        of (first token, tokens) on the device, or None when every token is a unit of its own)."""
        longest = 1 if ctx.fixed_shape else ctx.max_segment_len
        rows = ops.latent_attention_mma_rows(self.kv_rank, self.kv_rank + self.rot_dim, self.heads * longest)
        per = rows // self.heads
        if per <= 1 or longest == 1:
            return rows, None
        return rows, self._units(ctx, per)

    def _expanded(self, ctx):
        """None, or how the step's segments go through keys and values per head: (blocks [n, 2] and tiles [m, 4] on the device, see
        `ops.latent_keys_values` and `ops.latent_prefill`; query rows a CTA holds and runs of the other segments' tokens like `_rows_and_units` and
        those tokens' rows, None if there are no others)."""
        if self.w_kv is None or ctx.fixed_shape:
            return None
        key = ("latent expanded", self.window, self.heads, self.dim + self.vdim, self.kv_rank, self.rot_dim)
        if key not in ctx.memo:
            ctx.memo[key] = self._plan_expanded(ctx)
        return ctx.memo[key]

    def _saved(self, tokens, pos0, keys):
        """About how many microseconds of kernels a portion saves through keys and values per head."""
        seen = tokens * pos0 + tokens * (tokens + 1) // 2
        if self.window is not None:
            seen = min(seen, tokens * self.window)
        make = self.heads * self.kv_rank * (self.dim + self.vdim)
        return (tokens * make / MAP_RATE + seen * self.heads * (2 * self.kv_rank + self.rot_dim) / LATENT_RATE
                - keys * make / MAKE_RATE - seen * self.heads * (self.dim + self.rot_dim + self.vdim) / PAIR_RATE)

    def _choose(self, starts, pos0s):
        """None, or which of a step's segments (first tokens, then the step's end; first positions) go through keys and values per head, as (segment, first
        token, one past its last, its position, first position of its blocks, their number), and the token ranges of the others."""
        lens = [b - a for a, b in zip(starts, starts[1:])]
        if max(lens, default=0) < EXPAND_MIN_TOKENS:
            return None
        room = EXPAND_MAX_BYTES // (2 * self.heads * (self.dim + self.vdim)) // 64

        def place(s, some, n):
            """Puts segment s at the end of `some`, which holds n blocks, if it may go there; the blocks it holds then."""
            a, b, pos0 = starts[s], starts[s + 1], pos0s[s]
            first = 0 if self.window is None else max(0, pos0 - self.window + 1) // 64 * 64
            own = (pos0 + b - a - first + 63) // 64
            if 64 * own > EXPAND_MAX_CONTEXT * (b - a) or n + own > room:
                return n
            some.append((s, a, b, pos0, first, own))
            return n + own

        some, n = [], 0
        for s, length in enumerate(lens):
            if length >= EXPAND_MIN_TOKENS:
                n = place(s, some, n)
        if not some:
            return None
        taken = {c[0] for c in some}
        rest = [s for s, length in enumerate(lens) if length and s not in taken]
        every = []
        for i, s in enumerate(rest):
            n = place(s, every, n)
            if len(every) == i:
                break
        if len(every) == len(rest):   # one form serves the whole step
            return some + every, []
        if sum(self._saved(c[2] - c[1], c[3], 64 * c[5]) for c in some) < EXPAND_BESIDE_SAVED_US:
            return None
        return some, [(starts[s], starts[s + 1]) for s in rest]

    def _plan_expanded(self, ctx):
        chosen = self._choose(ctx.h_seg_start.tolist(), ctx.h_seg_pos0.tolist())
        if chosen is None:
            return None
        some, rest = chosen
        tiles, spans, n_blocks = [], [], 0
        for s, a, b, pos0, first, n in some:
            tiles += [(t, min(128, b - t), pos0 + t - a, 64 * n_blocks - first) for t in range(a, b, 128)]
            spans.append((s, first, n_blocks, n_blocks + n))
            n_blocks += n
        tiles.sort(key=lambda t: -(t[2] + t[1] if self.window is None else min(t[2], self.window) + t[1]))   # the tiles that see the most keys first
        rows, runs, tokens = 0, [], []
        if rest:
            rows = ops.latent_attention_mma_rows(self.kv_rank, self.kv_rank + self.rot_dim, self.heads * max(b - a for a, b in rest))
            runs = _runs(rest, max(1, rows // self.heads))
            for a, b in rest:
                tokens += range(a, b)
        m, n = 4 * len(tiles), 4 * len(tiles) + 2 * n_blocks
        staging = torch.empty(n + len(runs) + len(tokens), dtype=torch.int32, pin_memory=True)
        h = staging.numpy()
        h[:m] = [v for t in tiles for v in t]
        blocks = h[m:n].reshape(-1, 2)
        for s, first, i, j in spans:
            blocks[i:j, 0], blocks[i:j, 1] = s, np.arange(first, first + 64 * (j - i), 64)
        h[n:] = runs + tokens
        dev = staging.to(ctx.rt.device, non_blocking=True)
        part = lambda at, rows, cols: dev.as_strided((rows, cols), (cols, 1), at)
        return part(m, n_blocks, 2), part(0, len(tiles), 4), (rows, part(n, len(runs) // 2, 2), dev[n + len(runs):]) if rest else None

    def _units(self, ctx, per):
        key = ("latent units", per)
        if key not in ctx.memo:
            starts = ctx.h_seg_start.tolist()
            runs = _runs(zip(starts, starts[1:]), per)
            staging = torch.empty(len(runs), dtype=torch.int32, pin_memory=True)
            staging.numpy()[:] = runs
            ctx.memo[key] = staging.to(ctx.rt.device, non_blocking=True).view(-1, 2)
        return ctx.memo[key]

    def _tensor_cores(self, rt) -> bool:
        how = rt.options.latent_attention
        if how == "generic" or rt.act_dtype != torch.bfloat16:
            return False
        fits = ops.latent_attention_mma_supports(self.kv_rank, self.kv_rank + self.rot_dim)
        if how == "mma" and not fits:
            raise ValueError(f"latent_attention = \"mma\" needs a latent and a rotated part that are multiples of 16 (up to 512 and 576 together), got {self.kv_rank} and {self.rot_dim}")
        return fits

    adds_to_residual = True   # the output projection may add to the residual stream in its epilogue

    def forward(self, ctx, h, cache, residual=None):
        rt, T, H, r, rot = ctx.rt, ctx.n_tokens, self.heads, self.kv_rank, self.rot_dim
        cos, sin = self.position.tables(ctx)
        qd = rt.linear(h, self.w_in)
        q_nope = rt.empty((T, H, self.dim))
        q_full = rt.empty((T, H, r + rot), torch.float32)
        gate = None
        if self.gate:   # the gates' columns are the last of the first product; their sigmoid waits for the product with Wuv
            gate = (qd, qd.shape[2] - H)
        if self.q_rank is None:
            if self.gate:
                raise NotImplementedError("an output gate is built for layers whose queries go through a latent")
            ops.latent_prepare(qd, self.c_norm, self.norm_eps, cos, sin, ctx.positions, ctx.seg_of_token, q_nope, q_full, cache, H, self.dim, rot, r,
                               self.own_kv, rt.status)
        else:
            cq = rt.empty((T, self.q_rank))
            ops.latent_down(qd, self.q_rank, self.q_norm, cq, self.c_norm, self.norm_eps, cos, sin, ctx.positions, ctx.seg_of_token, cache, r, rot, rt.status)
            ops.latent_prepare(rt.linear(cq, self.w_uq), None, self.norm_eps, cos, sin, ctx.positions, ctx.seg_of_token, q_nope, q_full, cache, H, self.dim, rot, r,
                               False, rt.status)
        plan = self._expanded(ctx)
        v = rt.empty((T, H, self.vdim))
        if plan is None or plan[2] is not None:   # the tokens whose queries go to the latents' space
            tc = rt.options.expert_gemm != "simt"   # (the per-head maps have the m16n8k16 kernel and the FMA kernel)
            only = None if plan is None else plan[2][2]
            ops.gemm_heads(q_nope, self.wuk_t, q_full, r, tensor_cores=tc and ops.rows_mma_fits(q_nope, self.wuk_t), rows=only)
            n_slices, slice_keys = self._slices(ctx, cache.c_view())
            scratch = None
            if n_slices > 1:
                skey = ("latent scratch", H, r, n_slices)
                if skey not in ctx.memo:
                    ctx.memo[skey] = (rt.empty((T * H * n_slices * r,), torch.float32), rt.empty((T * H * n_slices * 2,), torch.float32))
                scratch = ctx.memo[skey]
            u = rt.empty((T, H, r))
            if self._tensor_cores(rt):
                rows, units = self._rows_and_units(ctx) if plan is None else plan[2][:2]
                ops.latent_attention_mma(q_full, cache, ctx.positions, ctx.seg_of_token, units, self.scale, u, r, n_slices, slice_keys, scratch, rt.status, rows, window=self.window, sink=self.sink_dev)
            else:
                ops.latent_attention(q_full, cache, ctx.positions, ctx.seg_of_token, self.scale, u, r, n_slices, slice_keys, scratch, rt.status, window=self.window, sink=self.sink_dev)
            ops.gemm_heads(u, self.wuv, v, self.vdim, tensor_cores=tc and ops.rows_mma_fits(u, self.wuv), gate=gate, rows=only)
        if plan is not None:   # and those that see keys and values per head (their rows of v hold nothing yet)
            kv, part = ops.latent_keys_values(cache, plan[0], ctx.seg_start, ctx.seg_pos0, self.w_kv, r, rot, rt.status, self.window)
            ops.latent_prefill(q_nope, q_full, r, plan[1], kv, part, self.scale, v, rt.status, window=self.window, sink=self.sink_dev, gate=gate)
            rt.next_in_order(ctx)   # that kernel's CTAs hold an SM's tensor memory: no product may wait for it while the norm behind lets another one start
        return rt.linear(v.view(T, H * self.vdim), self.wo, add_to=residual)
