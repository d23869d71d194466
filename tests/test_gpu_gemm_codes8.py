"""Prefill GEMM on 8-bit weights: exact codes, f32 folds of the scale groups, whatever the size of the scales."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from conftest import record_parity
from oracle import ztvm_oracle as zo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,size", [
    (33, 128, 1536, 1.0), (64, 129, 1600, 1.0), (65, 2048, 2112, 1.0), (47, 1, 1664, 1.0), (33, 17, 6144, 1.0),    # token tiles, K shares, rows past N
    (129, 257, 1728, 1.0), (200, 3072, 2048, 1.0), (128, 1000, 6144, 1.0), (700, 136, 4160, 1.0),                  # SPR % 4 of 0 to 3, last slots of 1 to 4 blocks
    (257, 20001, 128, 1.0), (1000, 10000, 64, 1.0), (513, 20000, 192, 1.0), (330, 8200, 320, 1.0),                # fewer blocks than teams, and few more
    (40, 300, 1600, 2.0**-17), (40, 300, 1536, 2.0**12), (130, 300, 1728, 0.0),                                   # scales among f16's subnormals, weights past f16's largest, none
])
def test_codes(M, N, K, size, backend, dev, oracle_c):
    p = z.synth.projection(N, K, M=M, bits=8, seed=M + N, sigma_s=0.01 / 17)
    rng = np.random.default_rng(K)
    s, b = p["scales"].astype(np.float32), p["biases"].astype(np.float32)
    if size != 1.0:
        spread = size * 2.0 ** rng.integers(-3, 4, size=(N, 1))             # rows of different sizes
        s, b = s * spread * 17, b * spread
    s, b = s.astype(np.float16), b.astype(np.float16)
    x = p["x"] * np.float16(2.0**-8) if size > 1 else p["x"]
    y = dev.empty((M + 1, N), np.float16, fill=-77.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, 64, 8, 1, 0), y, dev.put(x), dev.put(s), dev.put(p["W"]), dev.put(b))
    got = dev.get(y)
    assert backend.ctx.device_errors() == 0 and (got[M:] == -77.0).all()
    rows = np.unique(np.concatenate([np.arange(min(N, 300)), np.arange(max(0, N - 300), N)]))
    ref = oracle_c.matmul_f64(x, p["W"][rows], s[rows], b[rows], 64, 8, True)
    got = got[:M][:, rows].astype(np.float64)
    assert np.isfinite(got).all() and np.abs(ref).max() < 65504
    record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
    mags = oracle_c.matmul_f64(np.abs(x), p["W"][rows], s[rows], np.abs(b[rows]), 64, 8, True)
    # one rounding to f16 (2^-11, absolute 2^-25) of f32 sums: the matrix unit drops bits below 2^-23 of the largest partial sum once per 16
    # products, the folds and the meetings of teams and K shares round three more times per 64 codes
    bound = 2.0**-11 * np.abs(ref) + 2.0**-25 + 1.001 * (K / 16 + 3 * K / 64 + 12) * 2.0**-23 * mags
    assert (np.abs(got - ref) <= bound).all()
