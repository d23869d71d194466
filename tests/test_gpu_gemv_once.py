"""Small batches over several K tiles whose sums meet once (8-bit codes from two rows on, 4-bit ones from five on): rows that are one block of rounds
on a CTA, and one tile more; a short last slice; token counts below a power of two, the paired form. Beside them what meets at every K tile: 4-bit codes
of few rows, 8-bit ones of one."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from conftest import record_parity
from oracle import ztvm_oracle as zo
from test_gpu_batch import f16_bound, f32_bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,N,K,M", [
    (8, 148 * 64, 2112, 3), (8, 148 * 64 + 1, 2112, 3),          # four tiles a CTA and five; seventeen slices, the last of one run
    (8, 148 * 32, 4160, 8), (8, 148 * 32 + 1, 4096, 5),          # two tiles and three, eight columns
    (8, 148 * 64, 4096, 4), (8, 148 * 64 + 1, 4096, 4), (8, 148 * 32, 4096, 8),     # whole aligned slices, four columns and eight
    (8, 20, 6144, 2), (8, 1003, 2176, 1),                        # one row on some CTAs
    (4, 148 * 64, 4160, 2), (4, 148 * 64 + 1, 4352, 2), (4, 148 * 32, 8256, 7), (4, 700, 12288, 8),
    (4, 148 * 32, 4352, 5), (4, 148 * 32 + 1, 4352, 5), (4, 148 * 32 + 1, 8192, 8),
])
def test_sums_that_meet_once(bits, N, K, M, backend, dev, oracle_c):
    p = z.synth.projection(N, K, M=M, bits=bits, seed=M + N, sigma_s=0.01 * 15 / (2**bits - 1))
    y = dev.empty((M + 1, N), np.float16, fill=-77.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, 64, bits, 1, 0), y, dev.put(p["x"]), dev.put(p["scales"]), dev.put(p["W"]), dev.put(p["biases"]))
    got = dev.get(y)
    assert (got[M:] == -77.0).all()
    rows = np.unique(np.concatenate([np.arange(min(N, 200)), np.arange(max(0, N - 200), N)]))    # both ends of N
    ref = oracle_c.matmul_f64(p["x"], p["W"][rows], p["scales"][rows], p["biases"][rows], 64, bits, True)
    got = got[:M][:, rows].astype(np.float64)
    assert np.isfinite(got).all()
    record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
    mags = oracle_c.matmul_f64(np.abs(p["x"]), p["W"][rows], p["scales"][rows], np.abs(p["biases"][rows]), 64, bits, True)
    assert (np.abs(got - ref) <= f16_bound(ref, mags, K)).all()


def test_paired_form_meets_once(backend, dev, oracle_c):
    D, F, M = 8192, 148 * 16, 8                                   # gate and up: two tiles a CTA
    p = z.synth.projection(2 * F, D, M=M, bits=4, seed=5, sigma_s=0.01)
    h = dev.empty((M, F), np.float16, fill=float("nan"))
    backend.ctx.fused_ffn(z.MmDesc(D, F, M, 64, 4, 1, 0), h, *[dev.put(p[k]) for k in ("x", "scales", "W", "biases")])
    some = np.unique(np.concatenate([np.arange(100), np.arange(F // 2, F // 2 + 40), np.arange(F - 100, F)]))
    both = np.concatenate([some, F + some])                       # gate rows, then their up rows
    W, s, b = p["W"][both], p["scales"][both], p["biases"][both]
    ref = zo.fused_ffn_f64(p["x"], W, s, b, len(some))
    mags = oracle_c.matmul_f64(np.abs(p["x"]), W, s, np.abs(b), 64, 4, True)
    y = oracle_c.matmul_f64(p["x"], W, s, b, 64, 4, True)
    g, u, eg, eu = y[:, :len(some)], y[:, len(some):], f32_bound(mags[:, :len(some)], D), f32_bound(mags[:, len(some):], D)
    silu = np.abs(g / (1 + np.exp(-g)))
    # f32 sums of gate and up through u * silu(g), whose slope in g is at most 1.1 |u|; expf, the division and the products in f32; one rounding to f16
    bound = 1.1 * (np.abs(u) + eu) * eg + silu * eu + (2.0**-11 + 2.0**-20) * np.abs(ref) + 2.0**-25
    got = dev.get(h)[:, some].astype(np.float64)
    record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
    assert (np.abs(got - ref) <= bound).all()
