"""One-row matmuls of a recorded step in one launch: whatever they read and overwrite of one another, replays give what the same
calls give as steps of one call each, bit for bit, and that is the oracle's result."""
import numpy as np
import pytest

import zero_tvm_b200 as z
from oracle import ztvm_oracle as zo
from zero_tvm_b200.backend import pod_args, resolve_matmul

pytestmark = pytest.mark.gpu

FORMATS = [(4, False), (4, True), (3, False), (8, False)]


class Step:
    """Recorded calls over named one-row buffers."""

    def __init__(self, backend, dev, rng, bits, symmetric):
        self.be, self.dev, self.rng, self.bits, self.sym = backend, dev, rng, bits, symmetric
        self.group = 32 if symmetric else 64
        self.rec, self.bufs, self.weights = z.recorder.DecodeRecorder(backend), {}, []

    def buf(self, name, n, dtype=np.float16, values=None):
        self.bufs[name] = self.dev.empty((1, n), dtype, fill=0.0)
        if values is not None:
            self.bufs[name].copy_(self.dev.put(values))
        return self.bufs[name]

    def matmul(self, y, x, n, k, f32=False):
        q, W, s, b = z.synth.make_weights(self.rng, n, k, bits=self.bits, group=self.group, sigma_s=0.01 * 15 / (2**self.bits - 1))
        keep = np.float16(10 / np.sqrt(k))                # results about as large as their inputs, however long the chain
        s, b = s * keep, None if self.sym else b * keep
        entry = "int8_affine_matvec" if self.bits == 8 else resolve_matmul(affine=not self.sym, K=k, q3=self.bits == 3, out_f32=f32)
        self.rec.dispatch(entry, [self.bufs[y], self.bufs[x], self.dev.put(s), self.dev.put(W), pod_args(k, n, bits=self.bits, group=self.group)]
                          + ([] if b is None else [self.dev.put(b)]))
        self.weights.append((y, x, q, s, b))

    def check(self, replays=3):
        """Results one by one, then replays of the captured step from the same buffers."""
        import torch
        torch.cuda.synchronize()
        start = {k: v.clone() for k, v in self.bufs.items()}

        def restore():
            for k, v in self.bufs.items():
                v.copy_(start[k])
            torch.cuda.synchronize()

        for fn, args, _ in self.rec._calls:            # one by one: steps of one call
            self.be.ctx.step_begin(1)
            fn(*args, stream=1)
            self.be.ctx.step_end()
        torch.cuda.synchronize()
        want = {k: v.clone() for k, v in self.bufs.items()}
        restore()
        step = self.rec.capture()
        for _ in range(replays):
            restore()
            step.replay()
            torch.cuda.synchronize()
            for k, v in self.bufs.items():
                assert torch.equal(v, want[k]) and torch.isfinite(v.float()).all(), k
        assert self.be.ctx.device_errors() == 0
        return want

    def against_oracle(self, want, y):
        """Result buffer `y`, whose x no later call overwrote. f32 sums over exact codes: each of K terms rounds at 2^-24 of the
        largest partial sum, far below the f16 store's 2^-11; graded as the other GEMV tests are."""
        _, x, q, s, b = next(w for w in self.weights if w[0] == y)
        w32 = zo.dequant_w32(q, s, b, self.group, affine=b is not None)
        ref = want[x].cpu().numpy().astype(np.float64) @ w32.astype(np.float64).T
        got = want[y].cpu().numpy().astype(np.float64)
        assert zo.rel_err_scaled(got, ref, 1e-3) < 2e-3, y


@pytest.mark.parametrize("bits,symmetric", FORMATS)
@pytest.mark.parametrize("d,wide", [(64, 149), (192, 1), (320, 2368), (1024, 40), (2112, 320), (4160, 704)])
def test_reads_and_overwrites(bits, symmetric, d, wide, backend, dev):
    """Results read by the next call and by one further on, a buffer overwritten after it was read, one written twice; results of
    one row, of fewer rows than SMs, and tiles that end anywhere."""
    rng = np.random.default_rng(d + wide + bits)
    st = Step(backend, dev, rng, bits, symmetric)
    for name in ("a", "b", "c"):
        st.buf(name, d, values=z.synth.make_x(rng, 1, d))
    st.buf("n", wide)
    st.buf("f", wide, np.float32)
    st.buf("a2", d)
    st.matmul("n", "a", wide, d)            # reads a
    st.matmul("b", "a", d, d)
    st.matmul("c", "b", d, d)               # reads the last result
    st.matmul("a2", "b", d, d)              # ... and once more
    st.matmul("b", "c", d, d)               # overwrites what two calls read
    st.matmul("b", "a2", d, d)              # ... and overwrites that
    if bits != 8:
        st.matmul("f", "b", wide, d, f32=True)
    want = st.check()
    for y in ("n",) if bits == 8 else ("n", "f"):
        st.against_oracle(want, y)


@pytest.mark.parametrize("bits,symmetric", FORMATS)
@pytest.mark.parametrize("hidden,ffn", [(256, 8), (448, 1096), (1088, 2240)])
def test_activation_behind_a_matmul(bits, symmetric, hidden, ffn, backend, dev):
    """SiLU * up joins the matmul it reads, writes both buffers, and is waited for; where it reads something else it runs alone."""
    rng = np.random.default_rng(hidden + bits)
    st = Step(backend, dev, rng, bits, symmetric)
    down = ffn // 64 * 64
    st.buf("x", hidden, values=z.synth.make_x(rng, 1, hidden))
    for name, n in (("gu", 2 * ffn), ("h", ffn), ("gu2", 2 * ffn), ("h2", ffn), ("y", hidden), ("y2", hidden)):
        st.buf(name, n)
    for gu, h, y in (("gu", "h", "y"), ("gu2", "h2", "y2")):
        st.matmul(gu, "x", 2 * ffn, hidden)
        if gu == "gu2":
            st.matmul("y2", "x", hidden, hidden)          # between the two
        st.rec.silu_mul(st.bufs[h], st.bufs[gu], 1, ffn)
        if down:
            st.bufs[h + "_k"] = st.bufs[h][:, :down]
            st.matmul(y, h + "_k", hidden, down)
    want = st.check()
    st.against_oracle(want, "gu")
    if down:
        st.against_oracle(want, "y")


def test_more_calls_than_one_launch_takes_and_formats_in_turn(backend, dev):
    rng = np.random.default_rng(1)
    st = Step(backend, dev, rng, 4, False)
    st.buf("v0", 256, values=z.synth.make_x(rng, 1, 256))
    for i in range(70):
        st.buf(f"v{i + 1}", 256)
        st.bits = 8 if 30 <= i < 33 else 4
        st.matmul(f"v{i + 1}", f"v{i}" if i % 4 else "v0", 256, 256)
        if i % 8 == 7:
            st.buf(f"w{i}", 512)
            st.buf(f"s{i}", 256)
            st.matmul(f"w{i}", "v0", 512, 256)
            st.rec.silu_mul(st.bufs[f"s{i}"], st.bufs[f"w{i}"], 1, 256)
            st.bufs[f"v{i + 1}"] = st.bufs[f"s{i}"]
    st.check(replays=2)


def test_a_wait_that_runs_out(dev, monkeypatch):
    """The limit of a step's waits is set so short that they expire: the step ends all the same and says so, every time, and calls that wait
    for nothing are right."""
    import time
    import torch
    monkeypatch.setenv("ZTVM_STEP_WAIT_CYCLES", "1")
    be = z.backend.CudaMatmulBackend(0)
    st = Step(be, dev, np.random.default_rng(4), 4, False)
    sizes = (8256, 64, 8256, 64)                           # (of 64 rows most CTAs have none: they wait while the others multiply)
    for i, n in enumerate(sizes):
        st.buf(f"v{i}", n, values=z.synth.make_x(st.rng, 1, n))
    for i in range(3):
        st.matmul(f"v{i + 1}", f"v{i}", sizes[i + 1], sizes[i])
    step = st.rec.capture()
    with pytest.raises(z.ZtvmError, match="code 11"):
        be.ctx.device_errors()
    t0 = time.perf_counter()
    for run in [step.replay] * 20 + [st.rec.run_eager] * 20:
        run()
        torch.cuda.synchronize()
        with pytest.raises(z.ZtvmError, match="code 11"):
            be.ctx.device_errors()
    assert time.perf_counter() - t0 < 2.0
    be.ctx.step_begin(1)
    fn, args, _ = st.rec._calls[0]
    fn(*args, stream=1)
    be.ctx.step_end()
    torch.cuda.synchronize()
    assert be.ctx.device_errors() == 0
    st.against_oracle({k: v.clone() for k, v in st.bufs.items()}, "v1")
    be.close()


@pytest.mark.parametrize("bits,symmetric", FORMATS)
def test_a_launch_per_call(bits, symmetric, backend, dev):
    """joined=False: what the same calls give one by one, bit for bit, replayed and eager."""
    import torch
    st = Step(backend, dev, np.random.default_rng(bits), bits, symmetric)
    for name, d in (("a", 1024), ("b", 1024), ("c", 320), ("d", 1024)):
        st.buf(name, d, values=z.synth.make_x(st.rng, 1, d))
    st.matmul("b", "a", 1024, 1024)
    st.matmul("c", "b", 320, 1024)
    st.matmul("d", "c", 1024, 320)
    for fn, args, _ in st.rec._calls:
        fn(*args, stream=1)
    torch.cuda.synchronize()
    want = {k: v.clone() for k, v in st.bufs.items()}
    step = st.rec.capture(joined=False)
    for run in (step.replay, step.run_eager):
        for name in ("b", "c", "d"):
            st.bufs[name].fill_(float("nan"))
        torch.cuda.synchronize()
        run()
        torch.cuda.synchronize()
        assert all(torch.equal(v, want[k]) for k, v in st.bufs.items())
    assert backend.ctx.device_errors() == 0


def test_two_captured_steps_replay_side_by_side(backend, dev):
    """Each captured step counts arrivals in words of its own."""
    import torch
    rng = np.random.default_rng(2)
    steps = []
    for _ in range(2):
        st = Step(backend, dev, rng, 4, False)
        for i in range(4):
            st.buf(f"v{i}", 512, values=z.synth.make_x(rng, 1, 512) * 0.1)
        for i in range(3):
            st.matmul(f"v{i + 1}", f"v{i}", 512, 512)
        steps.append((st, st.check(), st.rec.capture()))
    streams = [torch.cuda.Stream() for _ in steps]
    for _ in range(20):
        for s, (_, _, step) in zip(streams, steps):
            with torch.cuda.stream(s):
                step.replay()
    torch.cuda.synchronize()
    for st, want, _ in steps:
        assert all(torch.equal(v, want[k]) for k, v in st.bufs.items())
    assert backend.ctx.device_errors() == 0


@pytest.mark.parametrize("bits,symmetric", FORMATS)
def test_other_calls_inside_a_step(bits, symmetric, backend, dev, oracle_c):
    """A step on the context's own stream: calls that are made of a matmul have its result when they go on, and find what was called before
    them done."""
    import torch
    rng = np.random.default_rng(bits)
    K, N, group, ctx = 576, 300, 32 if symmetric else 64, backend.ctx
    W, s, b = z.synth.make_weights(rng, N, K, bits=bits, group=group, affine=not symmetric)[1:]
    W2, s2, b2 = z.synth.make_weights(rng, K, 320, bits=bits, group=group, affine=not symmetric)[1:]
    desc, feed = z.MmDesc(K, N, 1, group, bits, int(not symmetric), 0), z.MmDesc(320, K, 1, group, bits, int(not symmetric), 0)
    w = [dev.put(s), dev.put(W), None if symmetric else dev.put(b)]
    w2 = [dev.put(s2), dev.put(W2), None if symmetric else dev.put(b2)]
    xs = [z.synth.make_x(rng, 1, K) for _ in range(3)]
    want = [oracle_c.matmul_f64(x, W, s, b, group, bits, not symmetric) for x in xs]
    x0 = z.synth.make_x(rng, 1, 320)
    got = [np.full((1, N), 7, np.float16) for _ in range(2)]
    pinned = torch.full((1, N), 7, dtype=torch.float16).pin_memory()
    dx, d0, mid, y, h = dev.put(xs[2]), dev.put(x0), dev.empty((1, K), np.float16), dev.empty((1, N), np.float16), dev.empty((1, N // 2), np.float16, fill=0.0)
    ctx.step_begin()
    try:
        ctx.int4_matmul(desc, y, dx, *w)                       # held back
        ctx.int4_matmul_host(desc, got[0], xs[0], *w)
        ctx.int4_matmul(feed, mid, d0, *w2)                    # held back
        ctx.int4_matmul_host(desc, got[1], xs[1], *w)
        ctx.int4_matmul_host_async(desc, pinned, torch.from_numpy(xs[2]).pin_memory(), *w)
        ctx.host_wait()
        ctx.int4_matmul(desc, y, dx, *w)                       # held back
        ctx.fused_ffn(z.MmDesc(K, N // 2, 1, group, bits, int(not symmetric), 0), h, dx, *w)
    finally:
        ctx.step_end()
    ctx.sync()
    for out, ref in zip(got + [pinned.numpy(), dev.get(y)], want + [want[2]]):
        assert zo.rel_err_scaled(out.astype(np.float64), ref, 1e-3) < 2e-3
    assert zo.rel_err_scaled(dev.get(mid).astype(np.float64), oracle_c.matmul_f64(x0, W2, s2, b2, group, bits, not symmetric), 1e-3) < 2e-3
    gate, up = want[2][:, :N // 2], want[2][:, N // 2:]
    assert zo.rel_err_scaled(dev.get(h).astype(np.float64), up * gate / (1 + np.exp(-gate)), 1e-2) < 4e-3


@pytest.mark.parametrize("bits,K", [(4, 4096), (4, 4352), (4, 8448), (4, 12288), (4, 12544), (4, 16640), (3, 12544), (8, 12544), (8, 16640)])
def test_rows_of_several_pieces_a_thread(bits, K, backend, dev, oracle_c):
    """A thread takes up eight activations at a time, 4096 a round, three rounds ahead: either side of one round and of three, and one more. Bound as in
    test_small_activations_of_whole_3_bit_slices: f32 sums that the matrix unit truncates, and the rounding to f16."""
    rng = np.random.default_rng(K + bits)
    N = 200
    _, W, s, b = z.synth.make_weights(rng, N, K, bits=bits, sigma_s=0.01 * 15 / (2**bits - 1))
    x = z.synth.make_x(rng, 1, K)
    ref = oracle_c.matmul_f64(x, W, s, b, 64, bits, True)
    mags = oracle_c.matmul_f64(np.abs(x), W, s, np.abs(b), 64, bits, True)
    codes = oracle_c.matmul_f64(np.ones_like(x), W, s, np.zeros_like(b), 64, bits, True)
    args = [dev.put(x), dev.put(s), dev.put(W), dev.put(b)]
    ys = [dev.empty((1, N), np.float16, fill=9.0) for _ in range(3)]
    backend.ctx.step_begin()
    for y in ys:
        backend.ctx.int4_matmul(z.MmDesc(K, N, 1, 64, bits, 1, 0), y, *args)
    backend.ctx.step_end()
    backend.ctx.sync()
    for y in ys:
        got = dev.get(y).astype(np.float64)
        tiny = 2.0**-20 * codes if bits == 3 else 0.0          # 3-bit: an activation under a code's power of two
        assert (np.abs(got - ref) <= 2.0**-11 * np.abs(ref) + 2.0**-25 + tiny + 1.001 * (K / 16 + 3 * K / 64 + 20) * 2.0**-23 * mags).all()
