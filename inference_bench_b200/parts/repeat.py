"""Runs of layers that differ in their weights and their place in the cache only, in steps outside a graph.

Such a layer's kernels are the ones of the layer before with other addresses, but making them costs the host much more than launching them: every
wrapper checks its tensors, asks for an output buffer and works out a tile (about 16 us a kernel, of which the launch is 4). A short prompt portion's
kernels take less than that, so the step waits for the host. Here the calls of one layer are noted as it runs, and the layers after it repeat them
with their own weights and cache entry in the noted layer's buffers: everything is ordered by the stream, as it is when the allocator hands a freed
buffer to the next layer. A layer is repeated only after one whose input and output are alike (the first of a run may have nothing to add to the
stream yet), inside one step. Measured when bfloat16 layers went this way: 61 tokens behind 900 in eight layers of the 0.6B sizes 1,237 to 870 us a step (443 us
of it on the device), a call 5 us. Those are launched by one call a layer now (kernels/dense.py: 445 us); this form has the float32 layers and page
or head sizes that the tensor-core attention kernels do not take.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from ..kernels import lib as L
from ..kernels import ops


class Repeat:
    """The noted layer of a step. `run` repeats it for a layer with an equal key."""

    def __init__(self, key, block, cache, pending):
        self.key, self.weights, self.view = key, block.repeat_weights(), cache.c_view()
        self.pending_in, self.pending = pending, None
        self.held: list = []        # the layer's buffers
        self.calls: list = []       # (name, arguments)
        self.plan: Optional[list] = None

    def close(self, pending) -> bool:
        """The layer has run and left `pending`: whether it can be repeated. A contribution that is more than a tensor (behind a layer of another
        arrangement, with a norm or a constant of its own) is not one the next layer gets."""
        self.pending = pending
        a, b = self.pending_in, pending
        alike = a is b is None or isinstance(a, torch.Tensor) and isinstance(b, torch.Tensor) and a.shape == b.shape
        return alike and len(set(self.weights)) == len(self.weights)

    def _places(self) -> list:
        """[(name, arguments, [(place, number of what stands there)])]: the weights by number, then the cache view, its first row, and the contribution."""
        at = {p: i for i, p in enumerate(self.weights)}
        n = len(self.weights)
        if self.pending_in is not None:
            at[self.pending_in.data_ptr()] = n + 2
        out = []
        for name, args in self.calls:
            subs = []
            for place, a in enumerate(args):
                if isinstance(a, ops.PoolRow):
                    subs.append((place, n + 1))
                elif isinstance(a, int):
                    if a in at:
                        subs.append((place, at[a]))
                elif getattr(a, "_obj", None) is self.view:
                    subs.append((place, n))
            out.append((name, list(args), subs))
        return out

    def run(self, block, cache):
        if self.plan is None:
            self.plan = self._places()
        new = block.repeat_weights()
        new += [C.byref(cache.c_view()), cache.tma()[1], self.pending.data_ptr() if self.pending is not None else None]
        for name, args, subs in self.plan:
            for place, i in subs:
                args[place] = new[i]
            L.call(name, *args)
        return self.pending
