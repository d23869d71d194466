"""GPU parity of the batched exact-code kernel (8-bit projections of more than eight rows, router logits of many tokens):
every tile shape of its dispatch, token counts and row counts around the tile edges, ragged K."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from oracle import ztvm_oracle as zo
from conftest import record_parity

pytestmark = pytest.mark.gpu


def f32_bound(magnitudes, K):
    """Largest error of the kernel's f32 sums: every partial sum is at most `magnitudes` = sum |x| (s q + |b|), the matrix
    unit drops bits below 2^-23 of it once per 16 products, the folds round three more times per 64 codes."""
    return (K / 16 + 3 * K / 64 + 4) * 2.0**-23 * magnitudes


def f16_bound(ref, magnitudes, K):
    """... plus one rounding to f16 (relative 2^-11, absolute 2^-25 below the normal range)."""
    return 2.0**-11 * np.abs(ref) + 2.0**-25 + 1.001 * f32_bound(magnitudes, K)


@pytest.mark.parametrize("M,N,K,f32", [
    # on 148 SMs: the tile whose busiest SM has the least to do
    (9, 257, 64, True), (32, 64, 192, False), (33, 65, 2112, False), (40, 19001, 128, False),    # 64 x 32 tiles, K split four ways
    (31, 65, 2112, False), (33, 65, 2112, True), (256, 9472, 256, True), (256, 9472, 192, False),  # (f16 results of more rows and work are the prefill GEMM's)
    (64, 18944, 320, True), (61, 18943, 320, False), (35, 18817, 64, True),     # 128 x 64 tiles: one wave of 148, 64 x 32 would be four
    (250, 9409, 192, True), (256, 9472, 256, False),                            # 128 x 128 tiles
])
def test_tile_shapes_8bit(M, N, K, f32, backend, dev, oracle_c):
    p = z.synth.projection(N, K, M=M, bits=8, seed=M + N, sigma_s=0.01 / 17)
    y = dev.empty((M + 1, N), np.float32 if f32 else np.float16, fill=-77.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, 64, 8, 1, int(f32)), y, dev.put(p["x"]), dev.put(p["scales"]), dev.put(p["W"]),
                            dev.put(p["biases"]))
    got = dev.get(y)
    assert (got[M:] == -77.0).all()
    rows = np.unique(np.concatenate([np.arange(min(N, 300)), np.arange(max(0, N - 300), N)]))    # both ends of N
    ref = oracle_c.matmul_f64(p["x"], p["W"][rows], p["scales"][rows], p["biases"][rows], 64, 8, True)
    got = got[:M][:, rows].astype(np.float64)
    assert np.isfinite(got).all()
    record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
    mags = oracle_c.matmul_f64(np.abs(p["x"]), p["W"][rows], p["scales"][rows], np.abs(p["biases"][rows]), 64, 8, True)
    assert (np.abs(got - ref) <= (f32_bound(mags, K) if f32 else f16_bound(ref, mags, K))).all()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("T,rows,D", [(9, 17, 64), (97, 257, 2048), (130, 129, 1472)])
def test_router_logits_many_tokens(bits, T, rows, D, backend, dev):
    rng = np.random.default_rng(T + rows + bits)
    x = z.synth.make_x(rng, T, D)
    _, W, s, b = z.synth.make_weights(rng, rows, D, bits=bits)
    logits = dev.empty((T, rows), np.float32, fill=float("nan"))
    backend.ctx.moe_router_logits(D, rows, T, bits, logits, dev.put(x), dev.put(W), dev.put(s), dev.put(b))
    got, ref = dev.get(logits), zo.router_logits_f64(x, W, s, b, bits)
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 1e-5 * np.sqrt(np.mean(ref * ref))


@pytest.mark.parametrize("bits,T,E,d,ffn,slots", [(3, 9, 40, 192, 72, 4), (3, 19, 40, 192, 72, 4), (3, 40, 12, 320, 136, 4), (3, 97, 3, 256, 200, 2),   # tiles of 16, 32, 64 pairs
                                                  (4, 33, 40, 192, 72, 4), (4, 20, 9, 448, 136, 4)])    # K the streaming kernel does not take
def test_grouped_experts(bits, T, E, d, ffn, slots, backend, dev, oracle_c):
    """Experts through the grouped form: rows that fill no 128-row block, K of 3, 5 and 4 scale groups, ragged
    last tiles, a skewed expert, gate (shared input) and down (input per slot)."""
    rng = np.random.default_rng(T + E)
    ids = rng.integers(0, E, size=(T, slots), dtype=np.uint32)
    ids[:, 0] = 1
    for N, K, per_slot in ((ffn, d, False), (d, 64 * ((ffn + 63) // 64), True)):
        _, W, s, b = z.synth.make_weights(rng, N, K, bits=bits, sigma_s=0.02, lead=(E,))
        x = z.synth.make_x(rng, T * slots if per_slot else T, K)
        y = dev.empty((T, slots, N), np.float16, fill=float("nan"))
        desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, bits, 1, 0), E, slots, T, K if per_slot else 0, N, slots * K if per_slot else K, slots * N, slots)
        backend.ctx.int4_matmul_moe(desc, y, dev.put(x), dev.put(s), dev.put(W), dev.put(b), dev.put(ids))
        got = dev.get(y)
        assert backend.ctx.device_errors() == 0 and np.isfinite(got).all()
        ref = oracle_c.moe_matmul_f64(x, W, s, b, ids, N, K, 64, bits, in_per_slot=per_slot)
        record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
        mags = oracle_c.moe_matmul_f64(np.abs(x), W, s, np.abs(b), ids, N, K, 64, bits, in_per_slot=per_slot)
        assert (np.abs(got - ref) <= f16_bound(ref, mags, K)).all()


@pytest.mark.parametrize("K", [64, 192, 320, 576, 896])
def test_tensor_memory_tiles_over_several_units_per_cta(K, dev, oracle_c, monkeypatch):
    """The f16-weight tiles with more units than two per SM and K of 1, 3, 5, 9 and 14 stages: the stages of a unit start on
    either parity, and the last packed slot holds one, two or three of them. Bound: the MMA's inputs are the oracle's own
    f16 weights, so only the f32 sums and the f16 result differ (f16_bound)."""
    monkeypatch.setenv("ZTVM_MOE_GROUPED", "1")
    be = z.backend.CudaMatmulBackend(0)
    E, T, N = 20, 1500, 2104
    rng = np.random.default_rng(K)
    ids = rng.integers(0, E, size=(T, 1), dtype=np.uint32)
    _, W, s, b = z.synth.make_weights(rng, N, K, bits=4, sigma_s=0.02, lead=(E,))
    x = z.synth.make_x(rng, T, K)
    y = dev.empty((T, 1, N), np.float16, fill=float("nan"))
    desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, 4, 1, 0), E, 1, T, 0, N, K, N, 1)
    be.ctx.int4_matmul_moe(desc, y, dev.put(x), dev.put(s), dev.put(W), dev.put(b), dev.put(ids))
    got = dev.get(y)
    assert be.ctx.device_errors() == 0 and np.isfinite(got).all()
    ref = oracle_c.moe_matmul_f64(x, W, s, b, ids, N, K, 64, 4, in_per_slot=False, w16=True)
    mags = oracle_c.moe_matmul_f64(np.abs(x), W, s, np.abs(b), ids, N, K, 64, 4, in_per_slot=False)
    assert (np.abs(got - ref) <= f16_bound(ref, mags, K)).all()
    be.close()
