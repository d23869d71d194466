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
