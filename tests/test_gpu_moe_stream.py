"""The streaming kernel of grouped experts where its split changes: one slice, three, five, nine and one per warp; rows that fill no
tile, outputs that share no word, chunks of one pair, and more chunks than a CTA looks up ahead. Bound: exact codes and f32 folds
(f16_bound)."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from conftest import record_parity
from oracle import ztvm_oracle as zo
from test_gpu_batch import f16_bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("K,N,E,T,slots,pad", [
    (256, 16, 9, 30, 3, 0),            # one slice: sixteen row groups, nobody to meet
    (256, 21, 7, 23, 3, 1),            # odd rows and odd output strides: single stores
    (512, 250, 20, 25, 4, 0),          # eight row groups of two
    (768, 33, 12, 20, 4, 0),           # three slices, a warp without work
    (1280, 40, 30, 40, 2, 0),          # five
    (2304, 24, 6, 13, 4, 0),           # nine
    (4096, 32, 4, 8, 4, 0),            # a slice for every warp
    (256, 16, 4, 8200, 4, 0),          # 4100 chunks, more than 24 on each CTA
])
def test_streamed_experts(bits, K, N, E, T, slots, pad, dev, oracle_c, monkeypatch):
    monkeypatch.setenv("ZTVM_MOE_GROUPED", "2")
    be = z.backend.CudaMatmulBackend(0)
    rng = np.random.default_rng(K + N)
    ids = rng.integers(0, E, size=(T, slots), dtype=np.uint32)
    ids[: T // 2, 0] = 1                                      # one expert of many chunks
    _, W, s, b = z.synth.make_weights(rng, N, K, bits=bits, sigma_s=0.02, lead=(E,))
    x = z.synth.make_x(rng, T, K)
    row = N + pad
    y = dev.empty((T, slots, row), np.float16, fill=7.0)
    desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, bits, 1, 0), E, slots, T, 0, row, K, slots * row, slots)
    be.ctx.int4_matmul_moe(desc, y, dev.put(x), dev.put(s), dev.put(W), dev.put(b), dev.put(ids))
    out = dev.get(y)
    assert be.ctx.device_errors() == 0
    got = out[..., :N]
    assert np.isfinite(got).all() and (out[..., N:] == 7.0).all()
    ref = oracle_c.moe_matmul_f64(x, W, s, b, ids, N, K, 64, bits, in_per_slot=False)
    record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
    mags = oracle_c.moe_matmul_f64(np.abs(x), W, s, np.abs(b), ids, N, K, 64, bits, in_per_slot=False)
    assert (np.abs(got - ref) <= f16_bound(ref, mags, K)).all()
    be.close()


@pytest.mark.parametrize("reuse", [False, True])
@pytest.mark.parametrize("d,ffn,E,T,slots", [
    (512, 256, 5, 11, 4), (512, 256, 5, 15, 3),          # one pair below nine per expert, and nine
    (2048, 256, 6, 9, 4), (256, 2048, 6, 9, 4),          # long and short K first: by itself the short one is batched, with a shared plan both go one way
    (1792, 512, 7, 12, 4), (2304, 512, 7, 12, 4),        # seven slices fill the warps, nine do not
    (1280, 640, 7, 12, 4), (320, 256, 7, 12, 4),         # one projection over whole slices, the other not: plans of two tile heights
    (512, 512, 3, 40, 2),                                # many pairs per expert: batched
])
def test_three_bit_experts_by_size(d, ffn, E, T, slots, reuse, dev, oracle_c):
    """The choice for 3-bit experts left to the library: both projections of a block over one id list, with a plan each and with one
    that they may share."""
    be = z.backend.CudaMatmulBackend(0)
    be.ctx.moe_plan_reuse(reuse)
    rng = np.random.default_rng(d + ffn + T)
    ids = rng.integers(0, E, size=(T, slots), dtype=np.uint32)
    ids_dev = dev.put(ids)
    for N, K, per_slot in ((ffn, d, False), (d, ffn, True)):
        _, W, s, b = z.synth.make_weights(rng, N, K, bits=3, sigma_s=0.02, lead=(E,))
        x = z.synth.make_x(rng, T * slots if per_slot else T, K)
        y = dev.empty((T, slots, N), np.float16, fill=float("nan"))
        desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, 3, 1, 0), E, slots, T, K if per_slot else 0, N, slots * K if per_slot else K, slots * N, slots)
        be.ctx.int4_matmul_moe(desc, y, dev.put(x), dev.put(s), dev.put(W), dev.put(b), ids_dev)
        got = dev.get(y)
        assert be.ctx.device_errors() == 0 and np.isfinite(got).all()
        ref = oracle_c.moe_matmul_f64(x, W, s, b, ids, N, K, 64, 3, in_per_slot=per_slot)
        record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
        mags = oracle_c.moe_matmul_f64(np.abs(x), W, s, np.abs(b), ids, N, K, 64, 3, in_per_slot=per_slot)
        assert (np.abs(got - ref) <= f16_bound(ref, mags, K)).all()
    be.close()
