"""Which consecutive calls of a recorded step may run side by side: the gate and up projections of an MoE block below the
pair counts at which such calls are grouped, and nothing that shares an output element or reads what the other writes."""
import pytest
import torch

import zero_tvm_b200 as z
from zero_tvm_b200.backend import moe_gate_pod_args
from zero_tvm_b200.recorder import DecodeRecorder, _independent_pair

E, D, FFN = 4, 512, 64


class FakeBackend:
    dispatch = dispatch_router_logits = staticmethod(lambda *a, **k: None)


def calls(tokens, slots, bits=4, up_out=None, up_ids=None, x=None, entry="int4_matmul_tiled_affine_moe"):
    be = FakeBackend()
    gu = torch.zeros(tokens, slots, 2 * FFN, dtype=torch.float16)
    x = torch.zeros(tokens, D, dtype=torch.float16) if x is None else x(gu)
    w = torch.zeros(E, FFN, D * bits // 32, dtype=torch.int32)
    s = torch.zeros(E, FFN, D // 64, dtype=torch.float16)
    ids = torch.zeros(tokens, slots, dtype=torch.int32)
    pod = moe_gate_pod_args(D, FFN, slots, bits)
    rec = DecodeRecorder(be)
    rec.dispatch(entry, [gu, x, s, w, pod, s, ids], (16, tokens, slots))
    out = gu.view(-1)[FFN:] if up_out is None else up_out(gu)
    rec.dispatch(entry, [out, x, s, w, pod, s, ids if up_ids is None else up_ids(ids)], (16, tokens, slots))
    return _independent_pair(be, *rec._calls)


@pytest.mark.parametrize("tokens,slots,bits,want", [(1, 9, 4, True), (7, 9, 4, True), (8, 8, 4, False), (1, 1, 4, True),
                                                    (1, 9, 3, True), (31, 1, 3, True), (4, 8, 3, False)])
def test_pairs_below_the_grouped_counts(tokens, slots, bits, want):
    entry = "int4_matmul_tiled_affine_q3_moe" if bits == 3 else "int4_matmul_tiled_affine_moe"
    assert calls(tokens, slots, bits, entry=entry) is want


def test_separate_outputs_may_run_side_by_side():
    assert calls(2, 3, up_out=lambda gu: torch.zeros(2 * gu.numel(), dtype=torch.float16)[gu.numel():])


@pytest.mark.parametrize("change", [
    dict(up_out=lambda gu: gu),                                     # the same elements
    dict(up_out=lambda gu: gu.view(-1)[FFN - 8:]),                  # eight elements of the first call's rows
    dict(up_out=lambda gu: gu.view(-1)[FFN + 8:]),                  # ... of its next row
    dict(up_ids=lambda ids: ids.clone()),                           # other experts
    dict(x=lambda gu: gu.view(-1)[:3 * D].view(3, D)),              # the first call writes the second one's activations
])
def test_overlapping_calls_stay_in_sequence(change):
    assert not calls(3, 4, **change)


class FakeStream:
    """Notes what a capture puts on it."""

    def __init__(self, name, log):
        self.cuda_stream, self.log = name, log

    def record_event(self):
        return self.cuda_stream

    def wait_event(self, event):
        self.log.append((self.cuda_stream, "waits for", event))


def recorded_token(be, tokens=1, slots=9):
    gu, x = torch.zeros(tokens, slots, 2 * FFN, dtype=torch.float16), torch.zeros(tokens, D, dtype=torch.float16)
    w, s = torch.zeros(E, FFN, D // 8, dtype=torch.int32), torch.zeros(E, FFN, D // 64, dtype=torch.float16)
    ids, pod = torch.zeros(tokens, slots, dtype=torch.int32), moe_gate_pod_args(D, FFN, slots)
    rec = DecodeRecorder(be)
    for out in (gu, gu.view(-1)[FFN:]):
        rec.dispatch("int4_matmul_tiled_affine_moe", [out, x, s, w, pod, s, ids], (16, tokens, slots))
    return rec


@pytest.mark.parametrize("plan,want", [
    (False, [("side", "waits for", "main"), ("main", "runs"), ("side", "runs"), ("main", "waits for", "side")]),
    (True, [("main", "runs"), ("main", "runs")]),
])
def test_calls_that_use_the_plan_are_captured_in_sequence(plan, want):
    """A context may group any number of pairs (its MoE kernel knob): only the library knows, and what shares its plan
    buffer must not become two branches."""
    log = []

    class Backend:
        def dispatch(self, entry, bindings, grid, stream=None):
            log.append((stream, "runs"))

        def uses_moe_plan(self, entry, bindings, grid):
            return plan

    recorded_token(Backend())._run_captured(FakeStream("main", log), FakeStream("side", log))
    assert log == want


@pytest.mark.parametrize("joined,want", [(True, ["begin", "runs", "runs", "end"]), (False, ["runs", "runs"])])
def test_steps_are_joined_unless_asked_otherwise(joined, want):
    log = []

    class Backend:
        class ctx:
            step_begin, step_end = staticmethod(lambda stream: log.append("begin")), staticmethod(lambda: log.append("end"))

        def dispatch(self, entry, bindings, grid, stream=None):
            log.append("runs")

        def uses_moe_plan(self, entry, bindings, grid):
            return True

    rec = recorded_token(Backend())
    rec._joined = joined
    rec._run_captured(FakeStream("main", log), FakeStream("side", log))
    assert log == want


@pytest.mark.gpu
@pytest.mark.parametrize("knob,tokens,want", [(None, 1, False), (None, 16, True), ("0", 64, False), ("1", 1, True), ("2", 1, True)])
def test_the_library_says_which_calls_use_the_plan(knob, tokens, want, dev, monkeypatch):
    if knob is None:
        monkeypatch.delenv("ZTVM_MOE_GROUPED", raising=False)
    else:
        monkeypatch.setenv("ZTVM_MOE_GROUPED", knob)
    be = z.backend.CudaMatmulBackend(0)
    for _, (entry, bindings, grid), _ in recorded_token(be, tokens)._calls:
        bindings = [t.cuda() if torch.is_tensor(t) and t.storage_offset() == 0 else torch.zeros(t.numel() + FFN, dtype=t.dtype, device="cuda")[FFN:]
                    if torch.is_tensor(t) else t for t in bindings]
        assert be.uses_moe_plan(entry, bindings, grid) is want
    be.close()


@pytest.mark.gpu
@pytest.mark.parametrize("knob", [None, "1", "2"])
def test_replayed_token_under_the_kernel_knob(knob, dev, monkeypatch):
    """Gate and up of one token, captured and replayed on other ids each time, give what plain launches give."""
    import numpy as np
    monkeypatch.setenv("ZTVM_MOE_GROUPED", knob) if knob else monkeypatch.delenv("ZTVM_MOE_GROUPED", raising=False)
    be = z.backend.CudaMatmulBackend(0)
    rng = np.random.default_rng(3)
    slots, (_, W, s, b) = 9, z.synth.make_weights(rng, FFN, D, bits=4, sigma_s=0.02, lead=(E,))
    x, gu = dev.put(z.synth.make_x(rng, 1, D)), dev.empty((1, slots, 2 * FFN), np.float16, fill=0.0)
    w, s, b = dev.put(W), dev.put(s), dev.put(b)
    ids, pod, rec = dev.empty((1, slots), np.uint32, fill=0), moe_gate_pod_args(D, FFN, slots), DecodeRecorder(be)
    for out in (gu, gu.view(-1)[FFN:]):
        rec.dispatch("int4_matmul_tiled_affine_moe", [out, x, s, w, pod, b, ids], (16, 1, slots))
    step = rec.capture()
    for k in range(4):
        ids.copy_(torch.tensor(rng.integers(0, E, (1, slots)).astype(np.int32)))
        gu.fill_(float("nan"))
        torch.cuda.synchronize()
        step.replay()
        torch.cuda.synchronize()
        got = gu.clone()
        gu.fill_(float("nan"))
        torch.cuda.synchronize()
        rec.run_eager()
        torch.cuda.synchronize()
        assert torch.equal(got, gu) and torch.isfinite(gu.float()).all()
    be.close()


@pytest.mark.gpu
@pytest.mark.parametrize("bits,E_,tokens,slots,K,N,shared,own", [
    (4, 64, 8, 8, 512, 64, True, False), (4, 64, 12, 8, 512, 64, True, True),       # K > N: from 3/2 pairs per expert on
    (4, 64, 8, 8, 192, 256, True, True), (4, 200, 16, 8, 512, 64, True, True),      # K < N; 128 pairs
    (4, 64, 7, 9, 192, 256, False, False),
    (3, 64, 8, 8, 512, 64, True, False), (3, 64, 9, 8, 512, 64, True, True), (3, 16, 10, 4, 512, 64, True, True),
    (3, 64, 8, 4, 64, 192, True, True), (3, 64, 8, 4, 128, 192, True, False), (3, 64, 10, 4, 128, 192, True, True), (3, 64, 31, 1, 64, 192, False, False),
])
def test_a_plan_of_one_call_needs_more_pairs(bits, E_, tokens, slots, K, N, shared, own, backend, dev):
    x, y = torch.zeros(tokens, K, dtype=torch.float16, device="cuda"), torch.zeros(tokens, slots, N, dtype=torch.float16, device="cuda")
    w, s = torch.zeros(E_, N, K * bits // 32, dtype=torch.int32, device="cuda"), torch.zeros(E_, N, K // 64, dtype=torch.float16, device="cuda")
    ids = torch.zeros(tokens, slots, dtype=torch.int32, device="cuda")
    desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, bits, 1, 0), E_, slots, tokens, 0, N, K, slots * N, slots)
    try:
        for reuse, want in ((True, shared), (False, own)):
            backend.ctx.moe_plan_reuse(reuse)
            assert backend.ctx.int4_matmul_moe_uses_plan(desc, y, x, s, w, s, ids) is want
    finally:
        backend.ctx.moe_plan_reuse(False)
