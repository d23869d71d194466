"""Prefill GEMM on 8-bit weights: two f16 terms per weight lose nothing that an f16 result shows, whatever the size of the scales."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from conftest import record_parity
from oracle import ztvm_oracle as zo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,size", [
    (33, 128, 64, 1.0), (64, 129, 576, 1.0), (65, 2048, 2112, 1.0), (33, 128, 1536, 1.0), (40, 300, 1600, 2.0**-17), (40, 300, 1536, 2.0**12), (130, 300, 1728, 0.0),        # tile widths, a last slot of one block, K shares in a cluster
    (128, 1000, 1152, 1.0), (129, 257, 320, 1.0), (200, 3072, 2048, 1.0), (256, 130, 192, 1.0), (257, 20001, 128, 1.0), (700, 136, 4160, 1.0),
    (40, 300, 512, 2.0**-17), (40, 300, 512, 2.0**13), (40, 300, 64, 0.0),   # scales among f16's subnormals, weights past f16's largest
])
def test_two_terms(M, N, K, size, backend, dev, oracle_c):
    """(Those of little work over a short K run on the kernel that multiplies the codes: the same bound.)"""
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
    # one rounding to f16 (2^-11, absolute 2^-25); the weight as f32 and its two terms 2^-22 of |s q + b| <= the terms of `mags`; the matrix
    # unit drops bits below 2^-23 of the largest partial sum once per 16 products, of either term; row bound 2^-39 of the row's largest
    # possible weight (255 s + |b|) per product
    top = np.max(255 * np.abs(s[rows].astype(np.float64)) + np.abs(b[rows].astype(np.float64)), axis=1)
    bound = 2.0**-11 * np.abs(ref) + 2.0**-25 + (2 * K / 16 + 6) * 2.0**-23 * mags + 2.0**-38 * top[None, :] * np.abs(x).astype(np.float64).sum(1)[:, None]
    assert (np.abs(got - ref) <= bound).all()
