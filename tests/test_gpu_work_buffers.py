"""The work buffers behind the grouped MoE matmul and the two-launch fused FFN: calls that may overlap -- on two streams,
in two captured graphs, in a graph and outside it -- never share one, a captured graph stays valid whatever the context
does afterwards, and a capture needs no call ahead of it."""
import numpy as np
import pytest

import zero_tvm_b200 as z

pytestmark = pytest.mark.gpu
E = 12


class Block:
    """One grouped matmul: bits, pairs and its own activations, ids and output."""

    def __init__(self, dev, bits, T, slots, seed, K=192, N=72):
        rng = np.random.default_rng(seed)
        _, W, s, b = z.synth.make_weights(rng, N, K, bits=bits, sigma_s=0.02, lead=(E,))
        self.args = [dev.put(z.synth.make_x(rng, T, K)), dev.put(s), dev.put(W), dev.put(b), dev.put(rng.integers(0, E, (T, slots), dtype=np.uint32))]
        self.y = dev.empty((T, slots, N), np.float16, fill=0.0)
        self.desc = z.MoeDesc(z.MmDesc(K, N, 1, 64, bits, 1, 0), E, slots, T, 0, N, K, slots * N, slots)

    def call(self, be, stream):
        be.ctx.int4_matmul_moe(self.desc, self.y, *self.args, stream=stream)

    def want(self, be):
        """The result of a call with nothing beside it."""
        import torch
        torch.cuda.synchronize()
        self.call(be, None)
        torch.cuda.synchronize()
        ref = self.y.clone()
        self.y.fill_(float("nan"))
        torch.cuda.synchronize()
        return ref


def captured(be, block, calls=1):
    import torch
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(calls):
            block.call(be, torch.cuda.current_stream())
    return g


@pytest.fixture
def fresh():
    be = z.backend.CudaMatmulBackend(0)
    yield be
    be.close()


# 4-bit from 64 pairs, 3-bit from 32 (both ran without a buffer once), 4-bit tiles, and a list beyond the one-block plan
SIZES = [(4, 9, 8), (3, 10, 4), (4, 40, 8), (4, 9000, 4)]


@pytest.mark.parametrize("bits,T,slots", SIZES)
def test_capture_needs_no_call_ahead(bits, T, slots, fresh, backend, dev):
    import torch
    blk = Block(dev, bits, T, slots, seed=T)
    ref = blk.want(backend)
    g = captured(fresh, blk)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(blk.y, ref)


def test_fused_ffn_capture_needs_no_call_ahead(fresh, backend, dev):
    import torch
    p = z.synth.projection(2 * 72, 192, M=20, seed=4)
    h, args = dev.empty((20, 72), np.float16, fill=float("nan")), [dev.put(p[k]) for k in ("x", "scales", "W", "biases")]
    desc = z.MmDesc(192, 72, 20, 64, 4, 1, 0)
    backend.ctx.fused_ffn(desc, h, *args)
    ref = torch.from_numpy(dev.get(h)).cuda()
    h.fill_(float("nan"))
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fresh.ctx.fused_ffn(desc, h, *args, stream=torch.cuda.current_stream())
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(h, ref)


@pytest.mark.parametrize("bits,T,slots", SIZES)
def test_a_graph_outlives_growth(bits, T, slots, fresh, dev):
    """A larger call after the capture, and plain calls between the replays, leave the graph's plan alone."""
    import torch
    blk, large = Block(dev, bits, T, slots, seed=T + 1), Block(dev, 4, 4 * T, 8, seed=T + 2)
    ref, ref_large = blk.want(fresh), large.want(fresh)
    g = captured(fresh, blk)
    for _ in range(3):
        large.y.fill_(float("nan"))
        blk.y.fill_(float("nan"))
        torch.cuda.synchronize()
        large.call(fresh, None)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(blk.y, ref) and torch.equal(large.y, ref_large)


@pytest.mark.parametrize("bits,T,slots", SIZES[:3])
def test_two_graphs_side_by_side(bits, T, slots, fresh, dev):
    import torch
    blocks = [Block(dev, bits, T, slots, seed=s) for s in (1, 2)]
    refs = [b.want(fresh) for b in blocks]
    graphs = [captured(fresh, b, calls=8) for b in blocks]
    streams = [torch.cuda.Stream() for _ in blocks]
    for _ in range(20):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(b.y, r) for b, r in zip(blocks, refs))


@pytest.mark.parametrize("bits,T,slots", SIZES[:3])
def test_streams_side_by_side(bits, T, slots, fresh, dev):
    """Six streams of one context: more than it keeps buffers for."""
    import torch
    blocks = [Block(dev, bits, T, slots, seed=s) for s in range(6)]
    refs = [b.want(fresh) for b in blocks]
    streams = [torch.cuda.Stream() for _ in blocks]
    for _ in range(20):
        for b, s in zip(blocks, streams):
            b.call(fresh, s)
    torch.cuda.synchronize()
    assert all(torch.equal(b.y, r) for b, r in zip(blocks, refs))


def test_buffers_of_dropped_graphs_are_taken_over(fresh, dev):
    """Captures of changing size, each dropped before the next: once the buffers that stay with their graphs are used up
    (64 MB), the device memory in use stays put. A pair takes 5.5 bytes of plan, so a capture here needs 5 to 17 MB."""
    import torch
    blocks = [Block(dev, 4, T, 8, seed=T, K=64, N=8) for T in (120000, 240000, 380000)]
    refs = [b.want(fresh) for b in blocks]

    def one(b, ref):
        g = captured(fresh, b)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(b.y, ref)

    for i in range(12):
        one(blocks[i % 3], refs[i % 3])
    before = torch.cuda.mem_get_info()[0]
    for i in range(18):
        one(blocks[i % 3], refs[i % 3])
    assert before - torch.cuda.mem_get_info()[0] < 16 << 20
