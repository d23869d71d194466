"""GPU parity of the prefill GEMM where its tiles and K shares can go wrong: every token tile (64, 128, 256, 352), one to eight
K shares (also uneven ones, and more shares than token blocks), scale groups of 32 (without biases and with:
two tables at the widest pitch, tiles of at most 256 tokens), 64 and 128 with rows off their 8- and
16-byte alignment (K = 64 x odd), rows past M, N that is no multiple of 8 or 128, f32 output."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from conftest import record_parity
from oracle import ztvm_oracle as zo
from test_gpu_gemm import FLOOR_FRAC, TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,affine", [(64, True), (32, False), (128, True), (32, True)])
@pytest.mark.parametrize("M,N,K,f32", [
    (17, 128, 128, False), (24, 40, 4096, False), (33, 3072, 1664, False), (64, 1000, 5120, True),      # 64-token tiles
    (65, 1001, 2176, False), (77, 2176, 3072, False), (128, 392, 8192, True),                           # 128
    (129, 250, 4224, False), (200, 5000, 1152, False), (257, 9600, 640, False), (300, 2048, 4096, False),  # 256, one to many shares
    (273, 12200, 1088, False), (700, 6200, 2176, True), (1000, 5900, 320, False), (352, 130, 4160, False),  # up to 352
    (65, 1696, 1152, False), (69, 1216, 1664, False), (390, 2338, 2112, False), (139, 1693, 2560, True), (130, 954, 4096, False),   # 128 in three and four
    (266, 2088, 5312, False), (259, 1692, 7232, False), (258, 2140, 4992, True),    # shares, 256 in two, five and eight, up to 352 in five, six and eight
    (1000, 6100, 1088, False), (300, 1003, 4096, True), (350, 20011, 128, False), (50, 20000, 1664, False), (260, 19900, 640, False),  # whole waves and a rest
])
def test_tiles_and_shares(group, affine, M, N, K, f32, backend, dev, oracle_c):
    if K % group:
        K += 64
    p = z.synth.projection(N, K, M=M, seed=M + N + K, group=group, affine=affine)
    y = dev.empty((M + 2, N), np.float32 if f32 else np.float16, fill=-77.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, group, 4, int(affine), int(f32)), y, dev.put(p["x"]), dev.put(p["scales"]),
                            dev.put(p["W"]), dev.put(p["biases"]) if affine else None)
    got = dev.get(y)
    assert backend.ctx.device_errors() == 0
    assert (got[M:] == -77.0).all()
    got = got[:M].astype(np.float64)
    ref = oracle_c.matmul_f64(p["x"], p["W"], p["scales"], p["biases"], group, 4, affine, w16=True)
    err = zo.rel_err_scaled(got, ref, FLOOR_FRAC)
    record_parity(err, zo.rel_err(got, ref))
    assert np.isfinite(got).all() and err <= TOL, err


@pytest.mark.parametrize("K", [192, 1088])
def test_odd_group_counts(K, backend, dev, oracle_c):
    """Rows of 3 and 17 groups of 64: every row's scales start at another offset inside their 8-byte word; tables that
    start 8 bytes into their allocation."""
    p = z.synth.projection(260, K, M=40, seed=K)
    s, b = (dev.put(np.concatenate([np.zeros(4, np.float16), p[t].reshape(-1)])) for t in ("scales", "biases"))
    y = dev.empty((40, 260), np.float16, fill=float("nan"))
    backend.ctx.int4_matmul(z.MmDesc(K, 260, 40, 64, 4, 1, 0), y, dev.put(p["x"]), s[4:], dev.put(p["W"]), b[4:])
    ref = oracle_c.matmul_f64(p["x"], p["W"], p["scales"], p["biases"], 64, 4, True, w16=True)
    assert backend.ctx.device_errors() == 0
    assert zo.rel_err_scaled(dev.get(y).astype(np.float64), ref, FLOOR_FRAC) <= TOL
