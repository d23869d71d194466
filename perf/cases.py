"""Timed workloads of the quantised matmul path: what an inference engine has this library do.

Three kinds of work, all through `CudaMatmulBackend` / `DecodeRecorder`:

  project  one projection of the dense path: one dispatch. The smallest call there is, and the unit that prefill is
           tuned by.
  layers   what a dense model's step dispatches: embedding rows, then per layer q|k|v, o, gate|up, SiLU * up and down,
           then the lm_head. m = 1 is a decode step, m = 2..8 the rows of a small batch or of a speculative draft
           being verified, larger m a chunk of a prompt (whose lm_head runs on the last row only).
  moe      a sparse model's FFN block per layer: router logits, top-k, gate, up, SiLU * up, down, weighted sum.

`recorded` steps are captured once by `DecodeRecorder` and replayed, the way an engine runs decode; the others issue
their dispatches one by one, the way it runs prompts, whose lengths differ from call to call.

Weight formats (`weights`), as checkpoints have them:
  mlx4  4-bit affine, groups of 64       mlx3  3-bit affine, groups of 64 (decode kernels only, dense and expert)
  mlx8  8-bit affine, groups of 64       mlc4  4-bit symmetric, groups of 32

Codes are uniform, scales |N(0, 0.01)| in units of a 4-bit code, biases N(0, 0.05), activations N(0, 1): the
distributions of `zero_tvm_b200.synth`, drawn on the device.
"""
from __future__ import annotations

import math

import torch

import zero_tvm_b200 as z
from zero_tvm_b200 import backend as zb
from zero_tvm_b200.recorder import DecodeRecorder

BITS = {"mlx4": 4, "mlx3": 3, "mlx8": 8, "mlc4": 4}
GROUP = {"mlx4": 64, "mlx3": 64, "mlx8": 64, "mlc4": 32}


def listed():
    dense = dict(kind="layers", hidden=4096, qkv=6144, ffn=12288, vocab=151936)
    sparse = dict(kind="moe", experts=256, hidden=2048, ffn=512, top_k=8, shared=True)
    return [
        # one decode projection, dispatched by itself: latency of a single small call
        dict(name="project decode", kind="project", weights="mlx4", n=8192, k=2048, m=1, recorded=False),
        # one prefill projection at the chunk length that prefill is quoted at
        dict(name="project prefill 512", kind="project", weights="mlx4", n=8192, k=2048, m=512, recorded=False),
        # one generated token of an 8B-class model (eight of its layers): the product's main loop, in each format
        # whose checkpoints decode this way
        dict(dense, name="decode mlx4", weights="mlx4", layers=8, m=1, recorded=True, fused=False),
        dict(dense, name="decode mlx3", weights="mlx3", layers=4, m=1, recorded=True, fused=False),
        dict(name="decode mlc4", kind="layers", hidden=3072, qkv=9216, ffn=8192, vocab=32064, weights="mlc4", layers=8,
             m=1, recorded=True, fused=False),
        # four rows at once (four sequences, or a draft of four tokens), dispatched call by call, FFN front half fused
        dict(dense, name="batch of 4 mlx4", weights="mlx4", layers=4, m=4, recorded=False, fused=True),
        # a full prompt chunk: the largest amount of arithmetic
        dict(dense, name="prompt chunk 1024 mlx4", weights="mlx4", layers=2, m=1024, recorded=False, fused=False),
        # a short prompt of ragged length on the symmetric format
        dict(name="short prompt 77 mlc4", kind="layers", hidden=3072, qkv=9216, ffn=8192, vocab=32064, weights="mlc4",
             layers=4, m=77, recorded=False, fused=False),
        # an ordinary prompt on an 8-bit checkpoint
        dict(name="prompt 200 mlx8", kind="layers", hidden=2048, qkv=3072, ffn=6144, vocab=151936, weights="mlx8",
             layers=2, m=200, recorded=False, fused=False),
        # one generated token of a sparse model (four of its FFN blocks)
        dict(sparse, name="moe decode mlx4", weights="mlx4", layers=4, m=1, recorded=True),
        # a prompt of ordinary length on a 3-bit sparse checkpoint
        dict(sparse, name="moe prompt 256 mlx3", weights="mlx3", layers=1, m=256, recorded=False),
        # a long prompt on a 4-bit sparse checkpoint
        dict(sparse, name="moe prompt 2048 mlx4", weights="mlx4", layers=1, m=2048, recorded=False),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A dimension of a model: whole scale groups, any number of them."""
    return 64 * max(lo // 64, min(hi // 64, _log_uniform(rng, lo, hi) // 64))


def _rows(rng):
    """Rows of a dense step: decode, a small batch, or a prompt of any length up to the chunk cap."""
    u = rng.random()
    return 1 if u < 0.35 else rng.randint(2, 8) if u < 0.55 else _log_uniform(rng, 9, 1024)


def draw(rng):
    kind = rng.choices(("project", "layers", "moe"), (2, 5, 3))[0]
    if kind == "moe":
        m = _log_uniform(rng, 1, 2048)
        return dict(kind=kind, experts=rng.randint(32, 256), hidden=_width(rng, 1024, 2880), ffn=_width(rng, 256, 1536),
                    top_k=rng.randint(2, 8), shared=rng.random() < 0.5, weights="mlx3" if rng.random() < 0.35 else "mlx4",
                    layers=2 if m <= 64 else 1, m=m, recorded=m <= 16)
    m = _rows(rng)
    weights = rng.choices(("mlx4", "mlc4", "mlx8", "mlx3"), (9, 4, 4, 3 if m == 1 else 0))[0]
    if kind == "project":
        # any number of output rows: a vocabulary or a shard of one is seldom a round number
        return dict(kind=kind, weights=weights, n=_log_uniform(rng, 512, 16384), k=_width(rng, 512, 12288), m=m,
                    recorded=False)
    hidden = _width(rng, 1024, 4096)
    recorded = m == 1 or (m <= 8 and rng.random() < 0.5)
    return dict(kind=kind, weights=weights, hidden=hidden, qkv=hidden + 256 * rng.randint(1, 8),
                ffn=64 * int(hidden * rng.uniform(2.0, 3.0) / 64), vocab=_log_uniform(rng, 32000, 151936),
                layers=4 if m <= 8 else 1, m=m, recorded=recorded,
                fused=m <= 8 and not recorded and weights in ("mlx4", "mlc4"))


# ---- inputs ---------------------------------------------------------------------------------------------------------
_backend = None


def _shared_backend():
    """One backend per process, as a program has one per GPU."""
    global _backend
    if _backend is None:
        _backend = zb.CudaMatmulBackend(torch.cuda.current_device())
    return _backend


class _Inputs:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def normal(self, *shape, sigma=1.0):
        return (torch.randn(shape, device="cuda", generator=self.g) * sigma).to(torch.float16)

    def matrix(self, fmt, n, k, *lead):
        """[packed codes, scales, biases or None] of `n` rows of length `k`, with leading stack axes."""
        bits = BITS[fmt]
        w = torch.randint(-2**31, 2**31 - 1, (*lead, n, k * bits // 32), dtype=torch.int32, device="cuda", generator=self.g)
        s = self.normal(*lead, n, k // GROUP[fmt], sigma=0.01 * 15 / (2**bits - 1)).abs()
        return w, s, None if fmt == "mlc4" else self.normal(*lead, n, k // GROUP[fmt], sigma=0.05)

    def ids(self, count, below):
        return torch.randint(0, below, (count,), dtype=torch.int32, device="cuda", generator=self.g)


def _empty(*shape, dtype=torch.float16):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _entry(fmt, k, m, f32=False):
    """The pipeline an engine picks for a projection of `m` rows."""
    affine = fmt != "mlc4"
    if fmt == "mlx8":
        return "int8_affine_matvec" if m == 1 else "int8_affine_batched"
    if m == 1:
        return zb.resolve_matmul(affine=affine, K=k, out_f32=f32, q3=fmt == "mlx3")
    if m <= 8:
        return "int4_matmul_batched_dyn" + ("_affine" if affine else "")
    return zb.pick_chunk_gemm(None, affine=affine, K=k)


class _State:
    """`calls`: (recorder method, backend method, arguments) of one pass; `outputs`: what they leave behind."""

    def __init__(self, case):
        self.case, self.calls, self.outputs, self.step, self.keep = case, [], {}, None, []

    def matmul(self, fmt, y, x, mat, k, n, m, f32=False):
        w, s, b = mat
        pod = zb.pod_args(k, n, bits=BITS[fmt], group=GROUP[fmt], m_rows=None if m == 1 else m)
        self.calls.append(("dispatch", "dispatch", (_entry(fmt, k, m, f32), [y, x, s, w, pod] + ([] if b is None else [b]))))

    def record(self, be):
        rec = DecodeRecorder(be)
        for name, _, args in self.calls:
            getattr(rec, name)(*args)
        self.step = rec.capture()


def _prepare_project(st, c, r):
    x = r.normal(c["m"], c["k"])
    y = _empty(c["m"], c["n"])
    st.matmul(c["weights"], y, x, r.matrix(c["weights"], c["n"], c["k"]), c["k"], c["n"], c["m"])
    st.outputs["y"] = y


def _prepare_layers(st, c, r):
    fmt, m, d, ffn = c["weights"], c["m"], c["hidden"], c["ffn"]
    head = r.matrix(fmt, c["vocab"], d)
    if fmt in ("mlx4", "mlx8"):        # the formats with an embedding kernel; the table is the lm_head's (tied)
        rows, ids = _empty(m, d), r.ids(m, c["vocab"])
        w, s, b = head
        entry = "embedding_affine_int8" if fmt == "mlx8" else "embedding_affine"
        st.calls.append(("embedding", "dispatch_embedding", (entry, [rows, ids, s, w, [m, 1], b], d)))
        st.outputs["embedded"] = rows
    for i in range(c["layers"]):
        x, attn, x2 = r.normal(m, d), r.normal(m, d), r.normal(m, d)   # normed inputs and the attention's output
        qkv, o, h, down = _empty(m, c["qkv"]), _empty(m, d), _empty(m, ffn), _empty(m, d)
        st.matmul(fmt, qkv, x, r.matrix(fmt, c["qkv"], d), d, c["qkv"], m)
        st.matmul(fmt, o, attn, r.matrix(fmt, d, d), d, d, m)
        gate_up = r.matrix(fmt, 2 * ffn, d)
        if c["fused"]:
            w, s, b = gate_up
            entry, more = ("fused_ffn", []) if b is None else ("fused_ffn_affine", [b])
            st.calls.append((None, "dispatch_fused_ffn", (entry, [h, x2, s, w, [ffn]] + more, d, ffn, m)))
        else:
            gu = _empty(m, 2 * ffn)
            st.matmul(fmt, gu, x2, gate_up, d, 2 * ffn, m)
            st.calls.append(("silu_mul", "silu_mul", (h, gu, m, ffn)))
        st.matmul(fmt, down, h, r.matrix(fmt, d, ffn), ffn, d, m)
        st.outputs.update({f"qkv{i}": qkv, f"o{i}": o, f"h{i}": h, f"down{i}": down})
    rows = m if m <= 8 else 1           # a prompt samples from its last row
    f32 = rows == 1 and fmt != "mlx8"   # the batched and the 8-bit kernels store f16
    logits = _empty(rows, c["vocab"], dtype=torch.float32 if f32 else torch.float16)
    st.matmul(fmt, logits, r.normal(rows, d), head, d, c["vocab"], rows, f32)
    st.outputs["logits"] = logits


def _prepare_moe(st, c, r):
    fmt, bits, T, E, d, ffn, K = c["weights"], BITS[c["weights"]], c["m"], c["experts"], c["hidden"], c["ffn"], c["top_k"]
    shared = c["shared"]
    slots, stack = zb.moe_slots(K, shared), E + int(shared)
    gate_entry = zb.resolve_matmul(affine=True, K=d, q3=fmt == "mlx3", moe=True)
    down_entry = zb.resolve_matmul(affine=True, K=ffn, q3=fmt == "mlx3", moe=True)
    for i in range(c["layers"]):
        x = r.normal(T, d)
        rw, rs, rb = r.matrix("mlx8", stack, d)                      # routers stay at 8 bits
        gate, up = r.matrix(fmt, ffn, d, stack), r.matrix(fmt, ffn, d, stack)
        down = r.matrix(fmt, d, ffn, stack)
        logits, scores = _empty(T, stack, dtype=torch.float32), _empty(T, slots, dtype=torch.float32)
        ids = _empty(T, slots, dtype=torch.int32)
        gu, h, y_slots, out = _empty(T, slots, 2 * ffn), _empty(T, slots, ffn), _empty(T, slots, d), _empty(T, d)
        gate_pod, down_pod = zb.moe_gate_pod_args(d, ffn, slots, bits), zb.moe_down_pod_args(d, ffn, slots, bits)
        st.calls += [
            ("router_logits", "dispatch_router_logits", ("moe_router_logits", [logits, x, rw, rs, rb, [d, stack]], (stack, T, 1))),
            ("router_topk", "moe_router_topk", (ids, scores, logits, E, K, True, shared, T)),
            ("dispatch", "dispatch", (gate_entry, [gu, x, gate[1], gate[0], gate_pod, gate[2], ids], (ffn // 4, T, slots))),
            ("dispatch", "dispatch", (gate_entry, [gu.view(-1)[ffn:], x, up[1], up[0], gate_pod, up[2], ids], (ffn // 4, T, slots))),
            ("silu_mul", "silu_mul", (h, gu, T * slots, ffn)),
            ("dispatch", "dispatch", (down_entry, [y_slots, h, down[1], down[0], down_pod, down[2], ids], (d // 4, T, slots))),
            ("moe_combine", "moe_combine", (out, y_slots, scores, T, slots, d)),
        ]
        st.outputs.update({f"ids{i}": ids, f"scores{i}": scores, f"y{i}": out})


def prepare(case, seed):
    be, st = _shared_backend(), _State(case)
    {"project": _prepare_project, "layers": _prepare_layers, "moe": _prepare_moe}[case["kind"]](st, case, _Inputs(seed))
    torch.cuda.synchronize()            # the library launches on its own stream: the inputs are complete before it does
    if case["recorded"]:
        st.record(be)
    else:
        st.bound = [(getattr(be, name), args) for _, name, args in st.calls]
    return st


def run(state):
    if state.step is not None:
        state.step.replay()
        return state.outputs
    if state.case["kind"] == "moe":
        _shared_backend().ctx.moe_plan_reuse(True)   # gate, up and down of a block share one plan
    for call, args in state.bound:
        call(*args)
    return state.outputs


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _matrix_bytes(fmt, n, k):
    return n * k * BITS[fmt] // 8 + (1 if fmt == "mlc4" else 2) * 2 * n * (k // GROUP[fmt])


def _matmul_work(fmt, n, k, m, out_bytes=2):
    """(bytes, flops): weights once, activations in, results out."""
    return _matrix_bytes(fmt, n, k) + 2 * m * k + out_bytes * m * n, 2 * m * n * k


def work(case):
    c = case
    m, fmt = c["m"], c["weights"]
    if c["kind"] == "project":
        parts = [_matmul_work(fmt, c["n"], c["k"], m)]
    elif c["kind"] == "layers":
        d, ffn = c["hidden"], c["ffn"]
        per_layer = [_matmul_work(fmt, c["qkv"], d, m), _matmul_work(fmt, d, d, m),
                     # gate, up and the activation can be one pass: h is all that has to leave it
                     (_matrix_bytes(fmt, 2 * ffn, d) + 2 * m * d + 2 * m * ffn, 2 * m * 2 * ffn * d),
                     _matmul_work(fmt, d, ffn, m)]
        rows = m if m <= 8 else 1
        parts = per_layer * c["layers"] + [_matmul_work(fmt, c["vocab"], d, rows, 4 if rows == 1 and fmt != "mlx8" else 2)]
        if fmt in ("mlx4", "mlx8"):
            parts.append((_matrix_bytes(fmt, m, d) + 2 * m * d, 2 * m * d))
    else:
        d, ffn, E, K = c["hidden"], c["ffn"], c["experts"], c["top_k"]
        slots, extra = K + int(c["shared"]), int(c["shared"])
        active = E * (1 - (1 - K / E) ** m) + extra        # experts that at least one of m tokens is routed to
        parts = [(_matrix_bytes("mlx8", E + extra, d) + active * (2 * _matrix_bytes(fmt, ffn, d) + _matrix_bytes(fmt, d, ffn))
                  + 2 * m * d + 2 * m * d + 8 * m * slots,
                  2 * m * (E + extra) * d + 2 * m * slots * 3 * d * ffn)] * c["layers"]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    """f16 results of f32 sums, over f32 weights or weights rounded to f16 (the matrix-unit paths): each rounding is
    2^-11 at most, a few of them in quadrature per value. Chains store f16 in between (h, and the expert outputs).
    Expert ids come from an ordering of f32 sums: two that differ in their last bits may swap."""
    if case["kind"] == "moe":
        return {"rel": 2e-3, "max": 0.05, "differ": 1e-3}
    return {"rel": 1e-3, "max": 0.02}
