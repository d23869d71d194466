"""A decode step as one CUDA graph: the engine records a fixed sequence of dispatches per token
(src/zero-tvm/engine-core.ts:2194-2202) and submits it as one command buffer; here the same sequence of calls through
the C ABI is captured once into a CUDA graph and replayed per token, so a step costs one launch on the host.

    rec = DecodeRecorder(backend)
    rec.dispatch("int4_matmul_sg_tiled_vec4h_affine", [qkv, x, s, W, pod, b], grid)   # any method of the backend
    rec.router_logits("moe_router_logits", [...], grid); rec.router_topk(...); ...
    step = rec.capture()        # one eager pass first (kernels loaded, bad calls rejected), then the capture
    step.replay()               # every buffer is bound by address, as in the engine's bind groups

Only calls of this library are recorded; whatever else a step needs (attention, norms) would be captured by its own
owner on the same stream. torch is the owner of the stream and the graph object (plumbing).
"""
from __future__ import annotations

from typing import Callable, List, Tuple

from .backend import _decode_matmul


def _span(buf):
    """Byte range of a bound buffer from its address on, or None where its size is unknown."""
    if hasattr(buf, "data_ptr"):
        return buf.data_ptr(), buf.data_ptr() + buf.numel() * buf.element_size()
    return None


def _independent_pair(be, a, b):
    """Whether two consecutive recorded calls are the gate and the up projection of one MoE block of a few pairs: same
    entry, PODArgs, activations, ids and grid, and outputs that share no element. (Whether the library runs them without
    the plan that calls of a context share is the library's to say: DecodeRecorder._side_by_side.)"""
    if a[0] != be.dispatch or b[0] != be.dispatch:
        return False
    (ea, ba, ga), (eb, bb, gb) = a[1], b[1]
    if ea != eb or ga != gb or len(ga) < 3 or len(ba) != 7 or len(bb) != 7 or list(ba[4]) != list(bb[4]):
        return False
    spans = [_span(t) for t in (ba[0], bb[0], ba[1], bb[1], ba[6], bb[6])]
    if None in spans or spans[2] != spans[3] or spans[4] != spans[5]:
        return False
    _, moe, desc = _decode_matmul(ea, ba[4])
    if not moe or desc is None or ga[1] * ga[2] >= (64 if desc[0].bits == 4 else 32):   # (more pairs fill the chip by themselves)
        return False
    rows, (_in_slot, out_slot, _in_tok, out_tok, _ids) = desc[0].N, desc[1]
    slots, tokens = ga[2], ga[1]
    lo, hi = sorted((spans[0][0], spans[1][0]))
    reach = 2 * ((tokens - 1) * out_tok + (slots - 1) * out_slot + rows)          # bytes from a call's first to its last element
    beside = rows * 2 <= hi - lo <= (out_slot - rows) * 2 and out_tok >= slots * out_slot   # rows of one in the gaps of the other
    if not (beside or hi - lo >= reach):
        return False
    return all(s[1] <= out or s[0] >= out + reach for s in (spans[2], spans[4]) for out in (lo, hi))   # neither writes what the other reads


class DecodeRecorder:
    def __init__(self, backend):
        self.be = backend
        self._calls: List[Tuple[Callable, tuple, dict]] = []
        self._graph = None
        self._stream = None
        self._joined = True

    # -- recording: the same surface as CudaMatmulBackend, minus the stream (the recorder owns it) --------------------
    def dispatch(self, entry, bindings, grid=(1, 1, 1)):
        self._calls.append((self.be.dispatch, (entry, list(bindings), tuple(grid)), {}))

    def router_logits(self, entry, bindings, grid=(1, 1, 1)):
        self._calls.append((self.be.dispatch_router_logits, (entry, list(bindings), tuple(grid)), {}))

    def embedding(self, entry, bindings, D):
        self._calls.append((self.be.dispatch_embedding, (entry, list(bindings), D), {}))

    def router_topk(self, ids, scores, logits, E, K, norm_topk, has_shared, tokens):
        self._calls.append((self.be.moe_router_topk, (ids, scores, logits, E, K, norm_topk, has_shared, tokens), {}))

    def silu_mul(self, out, gate_up, rows, ffn):
        self._calls.append((self.be.silu_mul, (out, gate_up, rows, ffn), {}))

    def moe_combine(self, out, y_slots, scores, tokens, slots, d):
        self._calls.append((self.be.moe_combine, (out, y_slots, scores, tokens, slots, d), {}))

    def __len__(self):
        return len(self._calls)

    def _side_by_side(self, a, b):
        """Two calls become branches of the graph only where the library runs both on the kernel that reads ids directly:
        the expert-sorted plan is one buffer, which the first call would fill while the second reads or fills it."""
        return _independent_pair(self.be, a, b) and not self.be.uses_moe_plan(*a[1]) and not self.be.uses_moe_plan(*b[1])

    def _run_captured(self, main, side):
        """The sequence inside the capture. The gate and up projections of a decoded token are a few CTAs each and read the
        same inputs: as two branches of the graph they run side by side (four blocks of one token, 256 experts of
        2048 x 512: 89 -> 73 us)."""
        i = 0
        while i < len(self._calls):
            if i + 1 < len(self._calls) and self._side_by_side(self._calls[i], self._calls[i + 1]):
                side.wait_event(main.record_event())
                fn, args, kw = self._calls[i]
                fn(*args, stream=main.cuda_stream, **kw)
                fn, args, kw = self._calls[i + 1]
                fn(*args, stream=side.cuda_stream, **kw)
                main.wait_event(side.record_event())
                i += 2
                continue
            # up to the next such pair: the library joins what it can into one launch
            end = i + 1
            while end < len(self._calls) and not (end + 1 < len(self._calls) and self._side_by_side(self._calls[end], self._calls[end + 1])):
                end += 1
            self._run_joined(main.cuda_stream, i, end)
            i = end

    def _run_joined(self, stream, first, last):
        """Calls first..last - 1 as one step: consecutive one-row matmuls become one launch (unless captured with joined=False)."""
        step_begin = getattr(getattr(self.be, "ctx", None), "step_begin", None) if self._joined else None
        if step_begin is None:
            for fn, args, kw in self._calls[first:last]:
                fn(*args, stream=stream, **kw)
            return
        step_begin(stream)
        try:
            for fn, args, kw in self._calls[first:last]:
                fn(*args, stream=stream, **kw)
        finally:
            self.be.ctx.step_end()

    def run_eager(self, stream=None):
        """The recorded sequence launched on `stream` (default: torch's current stream), joined as in the captured step."""
        import torch
        s = stream if stream is not None else torch.cuda.current_stream()
        self._run_joined(s.cuda_stream if s.cuda_stream else 1, 0, len(self._calls))

    def capture(self, plan_reuse: bool = True, joined: bool = True):
        """One eager pass (loads the kernels and sets their attributes; what it rejects is rejected before a
        capture), then the capture. plan_reuse: the MoE matmuls of the step share one expert-sorted plan per id list
        (valid because, inside the recorded sequence, only the recorded router writes the id list). joined: consecutive one-row
        matmuls become one launch, which starts when every SM is free of other work; False keeps a launch per call, for a step that
        must get on beside long kernels of other streams, or beside one that waits for something this step's stream does later.
        Results then are those of the same calls dispatched one by one, bit for bit."""
        import torch
        if not self._calls:
            raise ValueError("nothing recorded")
        self._joined = joined
        self._stream = torch.cuda.Stream()
        self._stream.wait_stream(torch.cuda.current_stream())
        self.be.ctx.moe_plan_reuse(plan_reuse)
        try:
            with torch.cuda.stream(self._stream):
                self._run_joined(self._stream.cuda_stream, 0, len(self._calls))
                self._stream.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=self._stream):
                    self.be.ctx.moe_plan_reuse(plan_reuse)          # drops any plan: the captured step builds its own
                    self._run_captured(self._stream, torch.cuda.Stream())
                self._stream.synchronize()
        finally:
            self.be.ctx.moe_plan_reuse(False)
        self._graph = g
        return self

    def replay(self):
        if self._graph is None:
            raise RuntimeError("capture() first")
        self._graph.replay()

    def synchronize(self):
        self._stream.synchronize()
