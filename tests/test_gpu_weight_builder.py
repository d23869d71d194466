"""Scales on both sides of every line of the f16 weight builder, read back bit for bit: |s| just below 2^-4 (codes as subnormals) and from there
on, subnormal and zero scales, biases inside and outside the guard, neighbouring groups on different paths. Through the hook, and through the
prefill GEMM and both expert tiles, whose activations are rows of the identity: a product with one and sums with zeros are exact, so every result
is the weight itself."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from oracle import ztvm_oracle as zo

pytestmark = pytest.mark.gpu
SCALES = [0x2BFF, 0xABFF, 0x2C00, 0xAC00, 0x2FFF, 0x3800, 0x0001, 0x8001, 0x03FF, 0x0400, 0x1000, 0x0000]
BIASES = [0x0000, 0x8000, 0x2A66, 0xB266, 0x3C00, 0x0003, 0x5640, 0xF000]
K, N = 256, 576


def weights(group, lead=()):
    """W, scales, biases: group g of row n has pair number `a` or (odd g) `b` of the 96, every pair beside six others."""
    pairs = np.array([(s, b) for s in SCALES for b in BIASES], dtype=np.uint16)
    n = np.arange(N)
    a, b = n % len(pairs), (37 * n + 11 * (n // len(pairs))) % len(pairs)
    take = np.where(np.arange(K // group) % 2 == 0, a[:, None], b[:, None])
    take = np.broadcast_to(take, (*lead, *take.shape))
    W = np.random.default_rng(group).integers(0, 2**32, size=(*lead, N, K // 8), dtype=np.uint32)
    return W, pairs[take, 0].view(np.float16), pairs[take, 1].view(np.float16)


def built(W, s, b, group):
    return zo.dequant_w16(zo.unpack_codes(W, 4), s, b, group, affine=b is not None)


@pytest.mark.parametrize("group,affine", [(64, True), (32, True), (128, True), (64, False), (32, False)])
def test_hook(group, affine, backend, dev):
    W, s, b = weights(group)
    b = b if affine else None
    out = dev.empty((N, K), np.float16, fill=float("nan"))
    backend.ctx.dequant(z.MmDesc(K, N, 1, group, 4, int(affine), 0), out, True, dev.put(s), dev.put(W), None if b is None else dev.put(b))
    want = built(W, s, b, group)
    assert np.isfinite(want.astype(np.float32)).all()
    assert np.array_equal(dev.get(out).view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("first,M", [(0, 256), (96, 64), (17, 100)])      # tiles of 256, 64 and 128 tokens
@pytest.mark.parametrize("group,affine", [(64, True), (32, True), (128, True), (64, False), (32, False)])
def test_prefill_gemm(group, affine, first, M, backend, dev):
    W, s, b = weights(group)
    b = b if affine else None
    y = dev.empty((M, N), np.float16, fill=float("nan"))
    x = np.eye(K, dtype=np.float16)[first:first + M]
    backend.ctx.int4_matmul(z.MmDesc(K, N, M, group, 4, int(affine), 0), y, dev.put(x), dev.put(s), dev.put(W), None if b is None else dev.put(b))
    got = dev.get(y)
    assert backend.ctx.device_errors() == 0
    assert np.array_equal(got.astype(np.float32), built(W, s, b, group).astype(np.float32).T[first:first + M])   # (zeros of either sign)


@pytest.mark.parametrize("tiles", ["ta", "sm"])
def test_expert_tiles(tiles, dev, monkeypatch):
    monkeypatch.setenv("ZTVM_MOE_GROUPED", "1")
    monkeypatch.setenv("ZTVM_MOE_TILES", tiles)
    be = z.backend.CudaMatmulBackend(0)
    W, s, b = weights(64, lead=(2,))
    ids = (np.arange(K, dtype=np.uint32) % 3 == 0).astype(np.uint32)[:, None]
    y = dev.empty((K, 1, N), np.float16, fill=float("nan"))
    desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, 4, 1, 0), 2, 1, K, 0, N, K, N, 1)
    be.ctx.int4_matmul_moe(desc, y, dev.put(np.eye(K, dtype=np.float16)), dev.put(s), dev.put(W), dev.put(b), dev.put(ids))
    got = dev.get(y)[:, 0].astype(np.float32)
    assert be.ctx.device_errors() == 0
    want = built(W.reshape(2 * N, -1), s.reshape(2 * N, -1), b.reshape(2 * N, -1), 64).astype(np.float32).reshape(2, N, K)
    assert np.array_equal(got, np.stack([want[int(ids[t, 0]), :, t] for t in range(K)]))
    be.close()
