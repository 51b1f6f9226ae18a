"""What calls keep to themselves: expert batches on several streams and in graphs beside direct calls."""
import time

import numpy as np
import pytest

from orome_b200 import synth

pytestmark = pytest.mark.gpu


class _Layer:
    """A layer of experts on the GPU, and calls with an input, activations and an output of their own."""

    def __init__(self, torch, F, E, H, M, seed):
        self.torch, self.F, self.E, self.H, self.M = torch, F, E, H, M
        parts = [synth.host_tensor(synth.Q4_K, E * M, H, seed=seed), synth.host_tensor(synth.Q4_K, E * M, H, seed=seed + 1),
                 synth.host_tensor(synth.Q5_K, E * H, M, seed=seed + 2)]
        self.mem = torch.from_numpy(np.concatenate(parts)).cuda()
        sg, sd = synth.tensor_bytes(synth.Q4_K, M, H), synth.tensor_bytes(synth.Q5_K, H, M)
        self.ref = F.ExpertLayerRef(self.mem.data_ptr(), F.ExpertProjRef(0, sg, synth.Q4_K), F.ExpertProjRef(E * sg, sg, synth.Q4_K),
                                    F.ExpertProjRef(2 * E * sg, sd, synth.Q5_K))

    def call(self, T, K, seed):
        t, rng = self.torch, np.random.default_rng(seed)
        idx, w = np.zeros((T, 8), np.int32), np.zeros((T, 8), np.float32)
        for i in range(T):
            idx[i, :K] = rng.permutation(self.E)[:K]
        w[:, :K] = rng.random((T, K))
        x = np.atleast_2d(synth.host_x(self.H, T, seed=seed))
        return {"T": T, "K": K, "x": t.from_numpy(x).cuda(), "idx": t.from_numpy(idx).cuda(), "w": t.from_numpy(w).cuda(),
                "act": t.empty((T, K, self.M), device="cuda"), "out": t.full((T, self.H), float("nan"), device="cuda")}

    def issue(self, ctx, c, stream):
        ctx.moe_ffn(self.ref, 0, c["x"].data_ptr(), c["T"], self.H, c["idx"].data_ptr(), c["w"].data_ptr(), c["K"], self.H, self.M,
                    c["act"].data_ptr(), c["out"].data_ptr(), self.H, stream)


@pytest.fixture()
def env():
    import torch
    from orome_b200 import format as F
    ctx = F.Context(0)
    yield torch, F, ctx
    torch.cuda.synchronize()
    assert ctx.status() == 0
    ctx.close()


def test_expert_batches_on_two_streams_of_a_context(env):
    """Same layer, same sizes, other tokens: whatever overlaps, each call gives the bits it gives alone."""
    torch, F, ctx = env
    layer = _Layer(torch, F, 8, 512, 512, 11)
    calls = [layer.call(200, 4, 21 + i) for i in range(2)]
    want = []
    for c in calls:
        layer.issue(ctx, c, 0)
        torch.cuda.synchronize()
        want.append(c["out"].clone())
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(30):
        for c in calls:
            c["out"].fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(3):
            for c, s in zip(calls, streams):
                layer.issue(ctx, c, s.cuda_stream)
        torch.cuda.synchronize()
        for c, w in zip(calls, want):
            assert torch.equal(c["out"], w)


def test_captured_expert_batches_own_their_scratch(env):
    """Graphs captured without any earlier call, replayed beside each other and beside a direct call; a graph that is gone gives
    its memory to the next capture."""
    torch, F, ctx = env
    layer = _Layer(torch, F, 8, 512, 512, 31)
    calls = [layer.call(200, 4, 41 + i) for i in range(4)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    graphs = []
    for mine in (calls[0:2], calls[2:3]):                  # two layers' worth in the first graph, one in the second
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            for c in mine:
                layer.issue(ctx, c, streams[0].cuda_stream)
        graphs.append(g)
    fresh = F.Context(0)
    want = []
    for c in calls:
        layer.issue(fresh, c, 0)
        torch.cuda.synchronize()
        want.append(c["out"].clone())
    for _ in range(20):
        for c in calls:
            c["out"].fill_(float("nan"))
        torch.cuda.synchronize()
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
        layer.issue(ctx, calls[3], streams[2].cuda_stream)
        torch.cuda.synchronize()
        for c, w in zip(calls, want):
            assert torch.equal(c["out"], w)
    del g, graphs
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    for _ in range(8):                                     # memory of one graph at a time
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            layer.issue(ctx, calls[0], streams[0].cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(calls[0]["out"], want[0])
        del g
        torch.cuda.synchronize()
        time.sleep(0.05)                                   # the driver tells of the graph's end from a thread of its own
    assert free - torch.cuda.mem_get_info(0)[0] <= 16 << 20      # eight pieces of 4 MiB would be 32
    fresh.close()


class _Product:
    """Y = X W^T with buffers of its own."""

    def __init__(self, torch, F, out_dim, in_dim, batch, seed, fmt=synth.Q4_K):
        self.out_dim, self.in_dim, self.batch = out_dim, in_dim, batch
        self.w = torch.from_numpy(synth.host_tensor(fmt, out_dim, in_dim, seed=seed)).cuda()
        self.ref = F.tensor_ref(self.w.data_ptr(), 0, fmt, out_dim, in_dim)
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        self.x = torch.randn(batch, in_dim, generator=g, device="cuda")
        self.y = torch.full((batch, out_dim), float("nan"), device="cuda")

    def issue(self, ctx, stream=0, batch=None):
        ctx.matvec(self.ref, self.x.data_ptr(), self.y.data_ptr(), batch or self.batch, self.in_dim, self.out_dim, stream)

    def error(self, torch, F, ctx):
        w = torch.empty(self.out_dim, self.in_dim, device="cuda")
        ctx.dequant_rows(self.ref, 0, self.out_dim, w.data_ptr())
        torch.cuda.synchronize()
        want = self.x.double() @ w.double().T
        return float((self.y.double() - want).norm() / want.norm())


TC_TOL = 5e-4          # fp16 operands


def test_captured_product_on_scratch_of_a_smaller_one(env):
    """Captured with room for a part of its packed X (two slices) and none for partial sums (whole tiles: no third launch a slice);
    then a larger direct call outgrows the scratch whose address the graph holds, and the graph is replayed."""
    torch, F, ctx = env
    small, p, big = _Product(torch, F, 256, 512, 16, 51), _Product(torch, F, 300, 8192, 2500, 52), _Product(torch, F, 256, 16384, 3000, 53)
    small.issue(ctx)
    torch.cuda.synchronize()
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    before = ctx.launch_count
    with torch.cuda.graph(g, stream=side):
        p.issue(ctx, side.cuda_stream)
    assert ctx.launch_count - before == 4
    big.issue(ctx)
    torch.cuda.synchronize()
    hold = [torch.full((1 << 20,), 7, dtype=torch.int32, device="cuda") for _ in range(32)]      # what a freed buffer would be given to
    for _ in range(2):
        p.y.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert p.error(torch, F, ctx) <= TC_TOL
    assert big.error(torch, F, ctx) <= TC_TOL and small.error(torch, F, ctx) <= TC_TOL
    assert all(int((h != 7).sum()) == 0 for h in hold)


def _device_bytes(torch, F, calls):
    """Device memory that the only context with scratch holds after `calls` (which have run before in another one: kernels are
    loaded, and torch has what it needs)."""
    held = []
    for _ in range(2):
        ctx = F.Context(0)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info(0)[0]
        calls(ctx)
        torch.cuda.synchronize()
        held.append(free - torch.cuda.mem_get_info(0)[0])
        ctx.close()
        torch.cuda.synchronize()
    return held[1]


def test_scratch_that_grows_is_no_larger_than_its_last_size(env):
    """Packed X of 2400, 3600 and 4096 vectors of 16384 (128 MiB at last; each kept and doubled: 225), and two partial tiles per
    pair of SMs (37 MiB); the pool takes memory 32 MiB at a time."""
    torch, F, _ = env
    p = _Product(torch, F, 512, 16384, 4096, 61)

    def calls(ctx):
        for b in (2400, 3600, 4096):
            p.issue(ctx, batch=b)
    assert _device_bytes(torch, F, calls) <= (128 + 37 + 2 * 32) << 20


def test_fixed_parts_of_a_long_prompt_bound_their_partial_sums(env):
    """OROME_OPT_TC_SPLIT = 12 on 512 vectors: the partial sums of 64 of them at a time, 24 MiB (all at once: 384 MiB)."""
    torch, F, _ = env
    p = _Product(torch, F, 8192, 4096, 512, 66, synth.Q8_0)

    def calls(ctx):
        ctx.set_option(F.OPT_TC_SPLIT, 12)
        p.issue(ctx)
        assert p.error(torch, F, ctx) <= TC_TOL
    assert _device_bytes(torch, F, calls) <= 96 << 20


def test_long_prompt_with_little_memory_left(env):
    """Packed X of 4096 vectors of 16384 takes 128 MiB; with less than that left the same product runs in smaller slices."""
    torch, F, _ = env
    p = _Product(torch, F, 256, 16384, 4096, 71)
    for b in (4096, 2048, 1024, 512):                      # every kernel that the slices may take is loaded
        warm = F.Context(0)
        p.issue(warm, batch=b)
        torch.cuda.synchronize()
        warm.close()
    ctx = env[2]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    p.y.fill_(float("nan"))
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info(0)[0] - (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        p.issue(ctx)
        torch.cuda.synchronize()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert p.error(torch, F, ctx) <= TC_TOL


def test_few_vectors_with_little_memory_left(env):
    """Room for the packed X, none for what only another form of the calls would use."""
    torch, F, ctx = env
    p, gate, up = _Product(torch, F, 1024, 4096, 8, 76), _Product(torch, F, 512, 1024, 8, 77), _Product(torch, F, 512, 1024, 8, 78)
    act = torch.full((8, 512), float("nan"), device="cuda")

    def calls(c):
        p.issue(c)
        c.gate_up_swiglu(gate.ref, up.ref, gate.x.data_ptr(), act.data_ptr(), 8, 1024, 512)
        torch.cuda.synchronize()
    warm = F.Context(0)
    calls(warm)                                            # every kernel is loaded
    want = p.y.clone(), act.clone()
    warm.close()
    p.y.fill_(float("nan"))
    act.fill_(float("nan"))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info(0)[0] - (48 << 20), dtype=torch.uint8, device="cuda")
    try:
        calls(ctx)
        calls(ctx)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert torch.equal(p.y, want[0]) and torch.equal(act, want[1])


def test_contexts_share_the_pool(env):
    """Scratch of a context that is gone serves the next one, and the last one gives everything back."""
    torch, F, ctx = env
    p, layer = _Product(torch, F, 512, 1024, 100, 81), _Layer(torch, F, 8, 512, 512, 82)
    c = layer.call(200, 4, 83)
    held = []
    for _ in range(3):
        a, b = F.Context(0), F.Context(0)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info(0)[0]
        for x in (a, b):
            p.issue(x)
            layer.issue(x, c, 0)
        a.close()
        p.issue(b)
        torch.cuda.synchronize()
        b.close()
        held.append(free - torch.cuda.mem_get_info(0)[0])
    assert max(held[1:]) <= 4 << 20
    assert p.error(torch, F, ctx) <= TC_TOL


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K])
def test_smaller_and_larger_batches_captured_after_a_warm_up_of_eight(env, fmt):
    """A token loop warms up once and captures its other batch sizes: what eight vectors leave behind (whichever form they took) serves a
    gate/up of two and of three, and 64 vectors of a product in as many launches as a direct call of them (tiles cut, sums added up)."""
    torch, F, ctx = env
    gate, up = (_Product(torch, F, 512, 1024, 8, s, fmt) for s in (91, 92))
    p = _Product(torch, F, 1024, 4096, 64, 93, fmt)
    act = torch.full((8, 512), float("nan"), device="cuda")

    def gate_up(c, batch, stream=0):
        c.gate_up_swiglu(gate.ref, up.ref, gate.x.data_ptr(), act.data_ptr(), batch, 1024, 512, stream)
    fresh = F.Context(0)
    want = []
    for b in (2, 3):
        gate_up(fresh, b)
        torch.cuda.synchronize()
        want.append(act[:b].clone())
    before = fresh.launch_count
    p.issue(fresh)
    direct = fresh.launch_count - before
    assert direct == 3                                     # pack, product, sums of cut tiles
    gate_up(ctx, 8)
    p.issue(ctx, batch=8)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for b, w in zip((2, 3), want):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            gate_up(ctx, b, side.cuda_stream)
        act.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(act[:b], w)
    before, g = ctx.launch_count, torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        p.issue(ctx, side.cuda_stream)
    assert ctx.launch_count - before == direct
    p.y.fill_(float("nan"))
    g.replay()
    torch.cuda.synchronize()
    assert p.error(torch, F, ctx) <= TC_TOL
    fresh.close()


def test_captured_gate_up_on_scratch_of_a_smaller_one(env):
    """2500 vectors of 8192 take 40 MiB of packed X, a first call leaves 32: captured, gate and up pack it in slices, each for itself.
    The bound: the same operands, but tiles that are not cut, 512 mma in a row that truncate at 2^-24 of a sum growing to its end, 512 / 3 *
    2^-24 = 1e-5 of a product on average; the activation is a product of two, and as much again for spread."""
    torch, F, ctx = env
    rows, batch, cols = 300, 2500, 8192
    first = [_Product(torch, F, rows, 256, batch, s) for s in (101, 102)]
    gate, up = (_Product(torch, F, rows, cols, batch, s) for s in (103, 104))
    act = torch.full((batch, rows), float("nan"), device="cuda")

    def gate_up(c, a, b, stream=0):
        c.gate_up_swiglu(a.ref, b.ref, a.x.data_ptr(), act.data_ptr(), batch, a.in_dim, rows, stream)
    gate_up(ctx, *first)                                   # room for both products' values
    torch.cuda.synchronize()
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    before = ctx.launch_count
    with torch.cuda.graph(g, stream=side):
        gate_up(ctx, gate, up, side.cuda_stream)
    assert ctx.launch_count - before >= 9                  # two slices of each: packing and product; the elementwise pass
    up.x = gate.x
    fresh = F.Context(0)
    for p in (gate, up):
        p.issue(fresh)
    torch.cuda.synchronize()
    want = torch.nn.functional.silu(gate.y.double()) * up.y.double()
    for _ in range(2):
        act.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert float((act.double() - want).norm() / want.norm()) <= 4e-5
    assert gate.error(torch, F, fresh) <= TC_TOL and up.error(torch, F, fresh) <= TC_TOL
    fresh.close()
