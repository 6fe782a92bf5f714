"""Layers of a dense decoder in bfloat16 steps with prompt portions, launched by one native call each (csrc/dense_layer.cu).

The parts make a layer's kernels one by one, each behind a wrapper that checks its tensors, asks for a buffer and works out a tile: about 15 us a kernel
on the host, which a short portion's kernels do not cover. Here the forms of the products, the index arrays and the buffers of a step are worked out
once, by the functions the parts use, and a layer brings its weights, its cache entry and what the layer before left to add. Same kernels, same order,
same arguments, so the same bits; the buffers belong to the step, and everything is ordered by the stream.
"""
from __future__ import annotations

import ctypes as C
import functools
from typing import Optional

import torch

from . import attention as A
from . import gemm_tcgen05 as G
from . import lib as L
from . import ops


class Product(C.Structure):
    """Mirror of IbDenseProduct in csrc/dense_layer.cu."""
    _fields_ = [("kind", C.c_int), ("bn", C.c_int), ("splits", C.c_int), ("wide", C.c_int)]


_p, _i, _f = C.c_void_p, C.c_int, C.c_float


class DenseStep(C.Structure):
    """Mirror of IbDenseStep."""
    _fields_ = ([(n, _p) for n in ("x", "h", "partial", "q", "o", "act", "part_o", "part_ml", "cos_t", "sin_t", "positions", "seg_of_token", "seg_start", "seg_pos0", "dec_tokens",
                                   "tile_seg", "tile_row0", "kv_map", "status", "stream")] + [(n, Product) for n in ("qkv", "out", "gate_up", "down")] +
                [(n, _i) for n in ("T", "hidden", "inter", "heads", "kv_heads", "head_dim", "rot_half", "window", "n_dec", "n_tiles", "max_slices", "tiles_per_slice", "tile_keys")] +
                [(n, _f) for n in ("norm_eps", "ff_norm_eps", "qk_eps", "scale")])


class DenseLayer(C.Structure):
    """Mirror of IbDenseLayer."""
    _fields_ = [(n, _p) for n in ("norm", "w_qkv", "w_out", "ff_norm", "w_gate_up", "w_down", "q_norm", "k_norm", "kv")] + [("kv_row0", C.c_longlong), ("delta", _p), ("delta_parts", _i)]


L.register("ib_dense_layer", [C.POINTER(DenseStep), C.POINTER(DenseLayer)])
L.register("ib_dense_sizes", [C.POINTER(_i), C.POINTER(_i)])


@functools.lru_cache(maxsize=1)
def _check_mirrors() -> None:
    """The library and the structures above are of one make."""
    step, layer = _i(), _i()
    L.load().ib_dense_sizes(C.byref(step), C.byref(layer))
    if (step.value, layer.value) != (C.sizeof(DenseStep), C.sizeof(DenseLayer)):
        raise L.KernelError(f"csrc/dense_layer.cu has structures of {step.value} and {layer.value} bytes, kernels/dense.py of {C.sizeof(DenseStep)} and {C.sizeof(DenseLayer)}")


# Steps of more tokens go layer by layer through the parts: their kernels take longer than the host, so nothing is gained (2,048 tokens in three layers of the
# 8B sizes already take 2,160 us either way), and one buffer for a whole layer's intermediates is harder for the allocator to find than its pieces (contexts of
# 8 requests built in steps of 8,192 tokens: 42 ms, 54 with it). Where between the two the line lies matters little; 2,048 tokens, the default portion,
# beside up to 512 decoded ones go this way.
MAX_TOKENS = 2560

KIND = {"single": 0, "pair": 1, "add": 2}
EPILOGUE = 3   # finished by the product's own epilogue


def _product(form: tuple) -> Product:
    return Product(KIND[form[0]], *form[1:]) if form[0] == "single" else Product(KIND[form[0]], 0, 1, 0)


def takes(ctx, cache) -> bool:
    """Whether this step's dense layers can go this way at all (their own sizes are asked in `DenseLayers`): a bfloat16 step with prompt portions on the
    kernels that TMA feeds, outside a layer whose calls are being noted."""
    opt = ctx.rt.options
    return (ctx.n_tokens <= MAX_TOKENS and ctx.rt.mode == "bfloat16" and ctx.rt.gemm != "simt" and not ctx.fixed_shape and ctx.n_segments != ctx.n_tokens and opt.prefill_attention != "tcgen05"
            and opt.decode_attention != "split" and L.notes.calls is None and cache.tma()[0] is not None)


class DenseLayers:
    """A step's dense layers of one key (`PreNormBlock.repeat_key`). `fits` tells whether the key's sizes are ones the kernels take."""

    def __init__(self, ctx, block, cache, x: torch.Tensor):
        _check_mirrors()
        m, f, rt, T = block.mixer, block.feed_forward, ctx.rt, ctx.n_tokens
        H, I, hd, opt = m.hidden, f.intermediate, m.head_dim, rt.options
        Q, R = m.heads * hd, (m.heads + 2 * m.kv_heads) * hd
        view = cache.c_view()
        cos, sin = m.position.tables(ctx)
        self.fits = (x.shape == (T, H) and x.dtype == torch.float32 and G.supports(H) and G.supports(Q) and G.supports(I) and hd == view.head_dim and m.kv_heads == view.kv_heads
                     and view.dtype == L.BF16 and A.has_tensor_core_kernel(torch.bfloat16, hd, m.heads, m.kv_heads) and (cos is None or cos.shape[0] == T))
        if not self.fits:
            return
        self.shapes = (R, H, H, Q, 2 * I, H, H, I)
        work = A._work_lists(ctx)
        rot_half = 0 if cos is None else cos.shape[1]
        if hd == 128 and rot_half in (0, 64) and G.qkv_in_epilogue(rt, T, R, H):
            qkv = Product(EPILOGUE, 0, 0, 0)
        else:
            qkv = _product(G.product_form(rt, T, R, H))
        out, down = _product(G.product_form(rt, T, H, Q, add=True)), _product(G.product_form(rt, T, H, I, add=True))
        if opt.swiglu_epilogue and G.swiglu_supported(T, H, I):
            bn, half = G.swiglu_form(T, I, opt.pair_min_tokens)
            gate_up = Product(EPILOGUE, bn, 0, 1 if half else 0)
        else:
            gate_up = _product(G.product_form(rt, T, 2 * I, H))
        max_slices = tps = 0
        if work["n_dec"]:
            tps = opt.stream_tiles_per_slice
            keys = work["max_pos"] + 1
            max_slices = -(-keys // (tps * A.decode_tile())) if tps else A.stream_slices(work["n_dec"], m.kv_heads, keys, rt.sm_count)
        # one buffer for all layers: h, the partial sums of whichever product ran last, then queries and attention output (the activation lies over
        # both: they are read for the last time before it is written), then the decoded tokens' slices
        self.partial_rows = max(p.splits * n for p, n in ((qkv, R), (out, H), (gate_up, 2 * I), (down, H)) if p.kind < 2) if min(p.kind for p in (qkv, out, gate_up, down)) < 2 else 0
        sizes = [2 * T * H, 4 * T * self.partial_rows, max(4 * T * Q, 2 * T * I), 4 * work["n_dec"] * m.heads * max_slices * hd, 8 * work["n_dec"] * m.heads * max_slices]
        ends, at = [], 0
        for n in sizes:
            ends.append(at)
            at += -(-n // 256) * 256
        self.buffer = rt.empty((at,), torch.uint8)
        base = self.buffer.data_ptr()
        h, partial, q, part_o, part_ml = (base + o for o in ends)
        self.partial, self.partial_at, self.T, self.H = partial, ends[1], T, H
        kv_map, _ = cache.tma()
        ptr = ops._ptr
        self.step = DenseStep(x.data_ptr(), h, partial, q, q + 2 * T * Q, q, part_o if work["n_dec"] else None, part_ml, ptr(cos), ptr(sin), ctx.positions.data_ptr(),
                              ctx.seg_of_token.data_ptr(), ctx.seg_start.data_ptr(), ctx.seg_pos0.data_ptr(), ptr(work["dec_tokens"]), ptr(work["tile_seg"]), ptr(work["tile_row0"]),
                              kv_map, rt.status.data_ptr(), ops._stream(), qkv, out, gate_up, down, T, H, I, m.heads, m.kv_heads, hd, rot_half, int(m.window or 0), work["n_dec"],
                              work["n_tiles"], max_slices, tps, work["tile_keys"], block.mixer_norm.eps, block.feed_forward_norm.eps, m.norm_eps, m.scale)
        self.left = down.splits if down.kind < 2 else 0   # partial sums the layers leave to add
        self._ref = C.byref(self.step)
        self.layer = DenseLayer()
        self._layer_ref = C.byref(self.layer)

    def run(self, block, cache, delta: Optional[int], parts: int) -> None:
        """One layer; delta, parts: address and number of the partial sums [T, hidden] that the layer before left to add."""
        m, f, l = block.mixer, block.feed_forward, self.layer
        if (m.wqkv.n, m.wqkv.k, m.wo.n, m.wo.k, f.wgu.n, f.wgu.k, f.wd.n, f.wd.k) != self.shapes:
            raise L.KernelError(f"a layer's matrices do not have the sizes of its key: {self.shapes}")
        l.norm, l.w_qkv, l.w_out = block.mixer_norm.w.data_ptr(), m.wqkv.weight.data_ptr(), m.wo.weight.data_ptr()
        l.ff_norm, l.w_gate_up, l.w_down = block.feed_forward_norm.w.data_ptr(), f.wgu.weight.data_ptr(), f.wd.weight.data_ptr()
        l.q_norm = None if m.q_norm is None else m.q_norm.data_ptr()
        l.k_norm = None if m.k_norm is None else m.k_norm.data_ptr()
        l.kv = C.addressof(cache.c_view())
        l.kv_row0, l.delta, l.delta_parts = cache.tma()[1], delta, parts
        if L.watched():
            self._one_by_one(C.byref(cache.c_view()))
        else:
            L.call_counted("ib_dense_layer", self._ref, self._layer_ref)

    def _one_by_one(self, kv) -> None:
        """The launches of `ib_dense_layer`, each through `call`, for somebody who looks at the calls: the same kernels on the same buffers."""
        s, l = self.step, self.layer
        T, H, I, Q = s.T, s.hidden, s.inter, s.heads * s.head_dim
        R, end = Q + 2 * s.kv_heads * s.head_dim, (s.status, s.stream)

        def product(p: Product, x, w, n: int, k: int) -> None:
            if p.kind == KIND["add"]:
                L.call("ib_gemm_tcgen05_2cta_add", x, w, s.x, T, n, k, *end)
            elif p.kind == KIND["pair"]:
                L.call("ib_gemm_tcgen05_2cta", x, w, s.partial, T, n, k, *end)
            else:
                L.call("ib_gemm_tcgen05", x, w, s.partial, T, n, k, p.bn, p.splits, p.wide, *end)

        def norm(delta, parts: int, w, eps: float) -> None:
            L.call("ib_add_rmsnorm", s.x, delta, parts if delta else 0, T * H if delta else 0, w, s.h, L.BF16, None, T, H, eps, 1, s.stream)

        norm(l.delta, l.delta_parts, l.norm, s.norm_eps)
        if s.qkv.kind == EPILOGUE:
            L.call("ib_gemm_qkv_tcgen05_2cta", s.h, l.w_qkv, T, H, l.q_norm, l.k_norm, s.qk_eps, s.cos_t, s.sin_t, s.positions, s.seg_of_token, s.q, kv, 1, s.heads, *end)
        else:
            product(s.qkv, s.h, l.w_qkv, R, H)
            L.call("ib_qk_norm_rope_kv", s.partial, s.qkv.splits, T * R, l.q_norm, l.k_norm, s.qk_eps, s.cos_t, s.sin_t, s.rot_half, s.positions, s.seg_of_token, s.q, L.BF16, kv, 1,
                   T, s.heads, s.status, None, s.head_dim, s.head_dim, 0, 0, 0, 0, 0, s.stream)
        if s.n_dec:
            L.call("ib_attention_decode_stream", s.q, kv, s.dec_tokens, s.n_dec, s.positions, s.seg_of_token, s.window, s.scale, s.part_o, s.part_ml, s.o, s.heads, s.max_slices,
                   s.tiles_per_slice, s.kv_map, l.kv_row0, *end)
        if s.n_tiles:
            L.call("ib_attention_prefill_ws", s.q, kv, s.tile_seg, s.tile_row0, s.n_tiles, s.seg_start, s.seg_pos0, s.window, s.scale, s.o, s.heads, s.kv_map, l.kv_row0, s.tile_keys,
                   *end)
        product(s.out, s.o, l.w_out, H, Q)
        norm(None if s.out.kind == KIND["add"] else s.partial, s.out.splits, l.ff_norm, s.ff_norm_eps)
        if s.gate_up.kind == EPILOGUE and s.gate_up.bn == 0:
            L.call("ib_gemm_swiglu_tcgen05_2cta", s.h, l.w_gate_up, s.act, T, I, H, None, 0.0, *end)
        elif s.gate_up.kind == EPILOGUE:
            L.call("ib_gemm_swiglu_tcgen05", s.h, l.w_gate_up, s.act, T, I, H, s.gate_up.bn, s.gate_up.wide, None, 0.0, *end)
        else:
            product(s.gate_up, s.h, l.w_gate_up, 2 * I, H)
            L.call("ib_silu_mul", s.partial, s.gate_up.splits, T * 2 * I, s.act, L.BF16, T, I, None, 0.0, s.stream)
        product(s.down, s.act, l.w_down, H, I)

    def pending(self) -> Optional[torch.Tensor]:
        """What the last layer left to add, as the parts hand it on."""
        if not self.left:
            return None
        n = self.left * self.T * self.H * 4
        return self.buffer[self.partial_at:self.partial_at + n].view(torch.float32).view(self.left, self.T, self.H)


class _NoLayers:
    fits = False


NO_LAYERS = _NoLayers()   # stands for a key whose layers the parts run
