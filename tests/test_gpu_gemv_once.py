"""Small batches over several K tiles whose sums meet once: rows that are one block of rounds on a CTA, and one tile more; a short last slice;
one row, token counts below a power of two, the paired form."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from conftest import record_parity
from oracle import ztvm_oracle as zo
from test_gpu_batch import f16_bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,N,K,M", [
    (8, 148 * 64, 2112, 3), (8, 148 * 64 + 1, 2112, 3),          # four tiles a CTA and five; seventeen slices, the last of one run
    (8, 148 * 32, 4160, 8), (8, 148 * 32 + 1, 4096, 5),          # two tiles and three, eight columns
    (8, 20, 6144, 2), (8, 1003, 2176, 1),                        # one row on some CTAs
    (4, 148 * 64, 4160, 2), (4, 148 * 64 + 1, 4352, 2), (4, 148 * 32, 8256, 7), (4, 700, 12288, 8),
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


def test_paired_form_meets_once(backend, dev):
    D, F, M = 8192, 148 * 16, 8                                   # gate and up: two tiles a CTA
    p = z.synth.projection(2 * F, D, M=M, bits=4, seed=5, sigma_s=0.01)
    h, gu = dev.empty((M, F), np.float16, fill=0.0), dev.empty((M, 2 * F), np.float16, fill=0.0)
    args = [dev.put(p[k]) for k in ("x", "scales", "W", "biases")]
    backend.ctx.fused_ffn(z.MmDesc(D, F, M, 64, 4, 1, 0), h, *args)
    backend.ctx.int4_matmul(z.MmDesc(D, 2 * F, M, 64, 4, 1, 0), gu, *args)
    g, u = (dev.get(gu)[:, i * F:(i + 1) * F].astype(np.float64) for i in (0, 1))
    want = u * g / (1 + np.exp(-g))
    # gate and up rounded to f16 once more on the right: a few half steps of each, through a slope of at most 1.1
    assert np.abs(dev.get(h) - want).max() <= 2.0**-9 * np.abs(u).max() * np.abs(g).max()
