"""GPU parity of the decode matmuls (1..8 rows) where their work split can go wrong: K tails of one to three runs,
odd numbers of scale groups (tables off their alignment), fewer items than warps, one row per CTA, several K tiles with
sums kept in shared memory, and the paired (fused FFN) form of every format."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from oracle import ztvm_oracle as zo
from conftest import record_parity
from test_gpu_batch import f16_bound, f32_bound

pytestmark = pytest.mark.gpu
FORMATS = {"w4": (4, 64, True), "w4sym": (4, 64, False), "g32": (4, 32, False), "g32affine": (4, 32, True), "w3": (3, 64, True), "w8": (8, 64, True)}


def magnitudes(p, oracle_c):
    """sum |x| (s q + |b|) per output (symmetric: b = -7 s), what the f32 error bound scales with."""
    b = np.abs(p["biases"]) if p["affine"] else (7 * p["scales"].astype(np.float32)).astype(np.float16)
    return oracle_c.matmul_f64(np.abs(p["x"]), p["W"], p["scales"], b, p["group"], p["bits"], True)


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("M,N,K,f32", [
    (1, 13, 64, False), (1, 150, 192, True), (2, 3000, 320, False), (1, 1184, 2112, False), (3, 37, 2368, True),
    (8, 301, 4160, False), (5, 40, 12288, True), (1, 24, 16384, False), (4, 2500, 256, True),
])
def test_shapes(fmt, M, N, K, f32, backend, dev, oracle_c):
    bits, group, affine = FORMATS[fmt]
    p = z.synth.projection(N, K, M=M, seed=M + N + K, bits=bits, group=group, affine=affine, sigma_s=0.01 if bits < 8 else 0.01 / 17)
    y = dev.empty((M + 1, N), np.float32 if f32 else np.float16, fill=-77.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, group, bits, int(affine), int(f32)), y, dev.put(p["x"]), dev.put(p["scales"]),
                            dev.put(p["W"]), dev.put(p["biases"]) if affine else None)
    got = dev.get(y)
    assert (got[M:] == -77.0).all()
    got = got[:M].astype(np.float64)
    ref = oracle_c.matmul_f64(p["x"], p["W"], p["scales"], p["biases"], group, bits, affine)
    assert np.isfinite(got).all()
    record_parity(zo.rel_err_scaled(got, ref, 1e-3), zo.rel_err(got, ref))
    mags = magnitudes(p, oracle_c)
    # groups of 32 fold twice as often per code: three more roundings per 32 codes
    assert (np.abs(got - ref) <= (2 * f32_bound(mags, K) if f32 else f16_bound(ref, 2 * mags, K))).all()


def test_tables_off_16_byte_alignment(backend, dev, oracle_c):
    """Scales that start 8 bytes into their allocation (all the ABI asks for) with groups of 32, whose items want 16."""
    p = z.synth.projection(200, 1024, M=1, seed=9, group=32, affine=False)
    s = dev.put(np.concatenate([np.zeros(4, np.float16), p["scales"].reshape(-1)]))
    y = dev.empty((1, 200), np.float16, fill=float("nan"))
    backend.ctx.int4_matmul(z.MmDesc(1024, 200, 1, 32, 4, 0, 0), y, dev.put(p["x"]), s[4:], dev.put(p["W"]), None)
    ref = oracle_c.matmul_f64(p["x"], p["W"], p["scales"], None, 32, 4, False)
    assert (np.abs(dev.get(y) - ref) <= f16_bound(ref, 2 * magnitudes(p, oracle_c), 1024)).all()


@pytest.mark.parametrize("fmt", ["g32", "w3", "w8", "w4"])
@pytest.mark.parametrize("ffn,K,M", [(9, 320, 1), (700, 2112, 3), (161, 4096, 8)])
def test_paired_form(fmt, ffn, K, M, backend, dev):
    bits, group, affine = FORMATS[fmt]
    p = z.synth.projection(2 * ffn, K, M=M, seed=ffn + K, bits=bits, group=group, affine=affine, sigma_s=0.01 if bits < 8 else 0.01 / 17)
    h = dev.empty((M + 1, ffn), np.float16, fill=-77.0)
    backend.ctx.fused_ffn(z.MmDesc(K, ffn, M, group, bits, int(affine), 0), h, dev.put(p["x"]), dev.put(p["scales"]), dev.put(p["W"]),
                          dev.put(p["biases"]) if affine else None)
    got = dev.get(h)
    assert (got[M:] == -77.0).all()
    ref = zo.fused_ffn_f64(p["x"], p["W"], p["scales"], p["biases"], ffn, group, bits, affine)
    err = zo.rel_err_scaled(got[:M].astype(np.float64), ref, 1e-3)
    record_parity(err, zo.rel_err(got[:M], ref))
    assert np.isfinite(got).all() and err <= 2e-3, err
