"""What f32 sums leave behind, seen through f16 results: rows whose exact results are zero."""
import numpy as np
import pytest

import zero_tvm_b200 as z

pytestmark = pytest.mark.gpu


def cancelling(seed, N, half, M, bits, group, symmetric):
    """x, W, s, b and the size of a result's terms (2-norm). The second half of K holds the products of the first, each group in another
    order and negated. Activations are mostly small beside a few large ones, as behind a SiLU * up."""
    rng = np.random.default_rng(seed)
    x1 = (rng.standard_normal((M, half)) ** 5 * 4).clip(-6e4, 6e4).astype(np.float16)
    q1 = rng.integers(0, 1 << bits, (N, half), dtype=np.uint8)
    order = np.concatenate([g * group + rng.permutation(group) for g in range(half // group)])
    s1 = np.abs(rng.standard_normal((N, half // group)) * 0.01 * 15 / (2**bits - 1)).astype(np.float16)
    b1 = (rng.standard_normal((N, half // group)) * 0.05).astype(np.float16)
    x, q = np.concatenate([x1, -x1[:, order]], 1), np.concatenate([q1, q1[:, order]], 1)
    s, b = np.concatenate([s1, s1], 1), None if symmetric else np.concatenate([b1, b1], 1)
    per = np.repeat(s.astype(np.float64), group, 1)
    terms = (per * q) ** 2 + ((7 * per) ** 2 if symmetric else np.repeat(b.astype(np.float64), group, 1) ** 2)
    return x, z.synth.pack_codes(q, bits), s, b, np.sqrt((x.astype(np.float64) ** 2 @ terms.T).mean())


@pytest.mark.parametrize("bits,symmetric,half,M", [
    (4, True, 1536, 1), (4, True, 4096, 1), (4, True, 160, 1), (4, True, 1056, 1),    # groups of 32: whole and ragged slices
    (8, False, 1024, 40), (8, False, 3072, 33), (8, False, 3072, 200), (8, False, 1088, 130),     # 8-bit prompts: token tiles, K shares
    (4, False, 1088, 1), (4, False, 320, 1), (4, False, 3648, 1), (3, False, 1088, 1), (3, False, 320, 1), (3, False, 3648, 1),    # K % 256
])
def test_sums_keep_f32(bits, symmetric, half, M, backend, dev):
    """Each result passes 2 K / group folds and a few more additions, each of which rounds by at most 2^-24 of a partial sum, evenly spread;
    a partial sum is about as large as the terms' 2-norm. By itself, and joined with another in a step."""
    group, N = 32 if symmetric else 64, 1100
    x, W, s, b, size = cancelling(half + M, N, half, M, bits, group, symmetric)
    K = 2 * half
    bound = np.sqrt((2 * K / group + 32) / 3) * 2.0**-24 * size + 2.0**-25                   # (f16 spacing near zero)
    args = [dev.put(x), dev.put(s), dev.put(W), None if b is None else dev.put(b)]
    desc = z.MmDesc(K, N, M, group, bits, int(not symmetric), 0)
    ys = [dev.empty((M, N), np.float16, fill=9.0) for _ in range(3)]
    backend.ctx.int4_matmul(desc, ys[0], *args)
    backend.ctx.step_begin()
    for y in ys[1:]:
        backend.ctx.int4_matmul(desc, y, *args)
    backend.ctx.step_end()
    backend.ctx.sync()
    for y in ys:
        err = np.sqrt((dev.get(y).astype(np.float64) ** 2).mean())
        assert err <= bound, (err / size, bound / size)


@pytest.mark.parametrize("M,N,K", [(200, 5000, 6144), (40, 25000, 4096)])
def test_sums_of_8_bit_prompts_lean_nowhere(M, N, K, backend, dev, oracle_c):
    """Sums that a matrix unit truncates over the whole of K come out too small. Here it has the 64 terms of a group, four truncations by 2^-24
    of a sum, and the rounding to f16, evenly spread within 2^-11, averages out: four standard deviations of a mean."""
    p = z.synth.projection(N, K, M=M, bits=8, seed=K, sigma_s=0.01 / 17)
    y = dev.empty((M, N), np.float16, fill=9.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, 64, 8, 1, 0), y, dev.put(p["x"]), dev.put(p["scales"]), dev.put(p["W"]), dev.put(p["biases"]))
    ref = oracle_c.matmul_f64(p["x"], p["W"], p["scales"], p["biases"], 64, 8, True)
    lean = (np.sign(ref) * (dev.get(y) - ref)).sum() / np.abs(ref).sum()
    assert abs(lean) <= 4 * 2.0**-24 + 4 * 2.0**-11 / np.sqrt(3 * M * N)


@pytest.mark.parametrize("K", [64, 320, 1600, 2112])
@pytest.mark.parametrize("size", [2.0**-10, 2.0**-14, 2.0**-20])
def test_small_activations_of_3_bit_rows(K, size, backend, dev, oracle_c):
    """K % 256 != 0: f32 activations whatever their size. One rounding to f16: 2^-11 of the result, 2^-25 among the subnormals."""
    rng = np.random.default_rng(K)
    N = 777
    _, W, s, b = z.synth.make_weights(rng, N, K, bits=3, sigma_s=0.02)
    x = (z.synth.make_x(rng, 1, K) * np.float32(size)).astype(np.float16)
    s, b = s * np.float16(8), b * np.float16(8)
    ref = oracle_c.matmul_f64(x, W, s, b, 64, 3, True)
    args = [dev.put(x), dev.put(s), dev.put(W), dev.put(b)]
    ys = [dev.empty((1, N), np.float16, fill=9.0) for _ in range(3)]
    backend.ctx.int4_matmul(z.MmDesc(K, N, 1, 64, 3, 1, 0), ys[0], *args)
    backend.ctx.step_begin()
    for y in ys[1:]:
        backend.ctx.int4_matmul(z.MmDesc(K, N, 1, 64, 3, 1, 0), y, *args)
    backend.ctx.step_end()
    backend.ctx.sync()
    for y in ys:
        got = dev.get(y).astype(np.float64)
        assert np.linalg.norm(got - ref) <= 2.0**-11 * np.linalg.norm(ref) + 2.0**-25 * np.sqrt(N)


@pytest.mark.parametrize("K", [256, 1536, 4352])
@pytest.mark.parametrize("size", [1.0, 2.0**-10, 2.0**-14])
def test_small_activations_of_whole_3_bit_slices(K, size, backend, dev, oracle_c):
    """K % 256 == 0: an activation under a code's power of two (1/32 at most) is f16 again, off by 2^-25 * 32 = 2^-20 where it falls among
    the subnormals; beside that, f32 sums that the matrix unit truncates, and the rounding to f16."""
    rng = np.random.default_rng(K)
    N = 333
    _, W, s, b = z.synth.make_weights(rng, N, K, bits=3, sigma_s=0.02)
    x = (z.synth.make_x(rng, 1, K) * np.float32(size)).astype(np.float16)
    ref = oracle_c.matmul_f64(x, W, s, b, 64, 3, True)
    mags = oracle_c.matmul_f64(np.abs(x), W, s, np.abs(b), 64, 3, True)
    codes = oracle_c.matmul_f64(np.ones_like(x), W, s, np.zeros_like(b), 64, 3, True)
    args = [dev.put(x), dev.put(s), dev.put(W), dev.put(b)]
    ys = [dev.empty((1, N), np.float16, fill=9.0) for _ in range(3)]
    backend.ctx.int4_matmul(z.MmDesc(K, N, 1, 64, 3, 1, 0), ys[0], *args)
    backend.ctx.step_begin()
    for y in ys[1:]:
        backend.ctx.int4_matmul(z.MmDesc(K, N, 1, 64, 3, 1, 0), y, *args)
    backend.ctx.step_end()
    backend.ctx.sync()
    for y in ys:
        got = dev.get(y).astype(np.float64)
        assert (np.abs(got - ref) <= 2.0**-11 * np.abs(ref) + 2.0**-25 + 1.001 * (2.0**-20 * codes + (K / 16 + 3 * K / 64 + 20) * 2.0**-23 * mags)).all()


@pytest.mark.parametrize("symmetric,N,K", [(False, 60000, 320), (False, 9000, 2112), (False, 1200, 9024), (True, 60000, 320), (True, 4096, 8192), (True, 1200, 9024)])
def test_single_rows_round_the_f32_result(symmetric, N, K, backend, dev):
    """4-bit rows of K % 256 != 0 or groups of 32 by themselves: one kernel whatever the result's type, so f16 results are the f32 ones rounded."""
    rng = np.random.default_rng(N + K)
    group = 32 if symmetric else 64
    _, W, s, b = z.synth.make_weights(rng, N, K, group=group, affine=not symmetric)
    args = [dev.put(z.synth.make_x(rng, 1, K)), dev.put(s), dev.put(W), None if symmetric else dev.put(b)]
    y16, y32 = dev.empty((1, N), np.float16, fill=9.0), dev.empty((1, N), np.float32, fill=9.0)
    backend.ctx.int4_matmul(z.MmDesc(K, N, 1, group, 4, int(not symmetric), 0), y16, *args)
    backend.ctx.int4_matmul(z.MmDesc(K, N, 1, group, 4, int(not symmetric), 1), y32, *args)
    backend.ctx.sync()
    assert (dev.get(y16) == dev.get(y32).astype(np.float16)).all()


@pytest.mark.parametrize("bits,symmetric,K,M", [(4, True, 320, 1), (4, False, 320, 1), (3, False, 320, 1), (8, False, 1600, 40)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 65504.0])
def test_activations_that_are_not_finite(bits, symmetric, K, M, value, backend, dev):
    """One such activation (or f16's largest) makes of a result what it makes of the f32 one: other kernels, the same folds."""
    group, N = 32 if symmetric else 64, 400
    rng = np.random.default_rng(K)
    _, W, s, b = z.synth.make_weights(rng, N, K, bits=bits, group=group, affine=not symmetric, sigma_s=0.01 * 15 / (2**bits - 1))
    x = z.synth.make_x(rng, M, K)
    x[M // 2, 77] = value
    args = [dev.put(x), dev.put(s), dev.put(W), None if symmetric else dev.put(b)]
    y32, ys = dev.empty((M, N), np.float32, fill=9.0), [dev.empty((M, N), np.float16, fill=9.0) for _ in range(2)]
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, group, bits, int(not symmetric), 1), y32, *args)
    backend.ctx.step_begin()
    for y in ys:
        backend.ctx.int4_matmul(z.MmDesc(K, N, M, group, bits, int(not symmetric), 0), y, *args)
    backend.ctx.step_end()
    backend.ctx.sync()
    want = dev.get(y32).astype(np.float64)
    for y in ys:
        got = dev.get(y).astype(np.float64)
        for kind in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(kind(got), kind(want)), kind
        ok = np.isfinite(want)
        assert np.allclose(got[ok], want[ok], rtol=2.0**-10, atol=2.0**-10 * np.abs(want[ok]).max(initial=0) / 16)
