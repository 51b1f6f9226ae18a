"""The batched form for few vectors (up to 32): plain and fused gate/up, against the fp64 oracle.  test_few_plan.py checks on the CPU that
all of these take this form, and which parts of it they reach.

Bound: x, the scales and minimums of a block and its weights are rounded to fp16 once (each 2^-11 / sqrt(3) * 0.74 = 2.1e-4 in the root
mean square, so 3 to 4.2e-4 of a product of many terms); 5e-4 asked of a product, as in the other batched form's tests, and twice
that of a fused one, which is a product of two.  A handful of outputs spreads more, since the terms of one may cancel where those of
many do not: their bound is eight times as wide.  A single vector's is three times, as in those tests: its rounding of x is common to
all of its outputs, so that it does not average out over them."""
import numpy as np
import pytest

import oracle
from orome_b200 import synth

pytestmark = pytest.mark.gpu

FORMATS = [(synth.Q8_0, 0), (synth.Q4_K, 0), (synth.Q4_K, 1), (synth.Q5_K, 0), (synth.Q5_K, 1), (synth.Q6_K, 0)]
# one row; a row tile and its neighbours; one tile a CTA and more; two passes of row tiles; 19 chunks that warps share unevenly, in more stages
# than the ring has
SHAPES = [(1, 512), (15, 256), (17, 768), (333, 2560), (2500, 512), (1003, 4864), (19200, 256)]
BATCHES = [4, 8, 9, 24, 32]
# rows, cols, vectors, fused: two passes of row tiles whose chunks (three, three and one; three and two) several warps share
PASSES = [(18951, 1792, 8, 0), (18951, 1280, 16, 0), (9501, 1792, 8, 1)]


@pytest.fixture(scope="module")
def env():
    import torch
    from orome_b200 import format as F
    ctx = F.Context(0)
    yield torch, F, ctx
    assert ctx.status() == 0
    ctx.close()


def _rel(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("fmt,variant", FORMATS)
@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("batch", BATCHES)
def test_few_vectors(env, fmt, variant, rows, cols, batch):
    torch, F, ctx = env
    ldx, ldy = cols + 4, rows + 3
    w = [synth.host_tensor(fmt, rows, cols, seed=s) for s in (rows, cols)]
    x = synth.host_x(cols, batch, seed=batch)
    wt = [torch.from_numpy(t).cuda() for t in w]
    xt = torch.full((batch, ldx), float("nan"), device="cuda")
    xt[:, :cols] = torch.from_numpy(x).cuda()
    y, act = (torch.full((batch, ldy), float("nan"), device="cuda") for _ in range(2))
    refs = [F.tensor_ref(t.data_ptr(), 0, fmt, rows, cols, variant) for t in wt]
    ctx.matvec(refs[0], xt.data_ptr(), y.data_ptr(), batch, ldx, ldy)
    ctx.gate_up_swiglu(refs[0], refs[1], xt.data_ptr(), act.data_ptr(), batch, ldx, ldy)
    torch.cuda.synchronize()
    gate, up = (oracle.matvec_f64(fmt, t, rows, cols, x, layout=variant).reshape(batch, rows) for t in w)
    few = 8 if rows * batch < 1000 else 1
    assert torch.isnan(y[:, rows:]).all() and torch.isnan(act[:, rows:]).all()
    assert _rel(y[:, :rows].cpu().numpy(), gate) <= 5e-4 * few
    assert _rel(act[:, :rows].cpu().numpy(), oracle.swiglu_f64(gate, up).reshape(batch, rows)) <= 1e-3 * few


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("rows,cols,batch,fused", PASSES)
def test_rows_in_two_passes(env, fmt, rows, cols, batch, fused):
    torch, F, ctx = env
    w = [synth.host_tensor(fmt, rows, cols, seed=s) for s in range(1 + fused)]
    x = synth.host_x(cols, batch, seed=batch)
    wt, xt = [torch.from_numpy(t).cuda() for t in w], torch.from_numpy(x).cuda()
    y = torch.full((batch, rows), float("nan"), device="cuda")
    refs = [F.tensor_ref(t.data_ptr(), 0, fmt, rows, cols) for t in wt]
    before = ctx.launch_count
    if fused:
        ctx.gate_up_swiglu(refs[0], refs[1], xt.data_ptr(), y.data_ptr(), batch, cols, rows)
    else:
        ctx.matvec(refs[0], xt.data_ptr(), y.data_ptr(), batch, cols, rows)
    assert ctx.launch_count - before == 2                  # the packing of X, the product
    torch.cuda.synchronize()
    want = [oracle.matvec_f64(fmt, t, rows, cols, x).reshape(batch, rows) for t in w]
    want, got = oracle.swiglu_f64(want[0], want[1]).reshape(batch, rows) if fused else want[0], y.cpu().numpy()
    bound = 1e-3 if fused else 5e-4
    assert _rel(got, want) <= bound
    assert max(_rel(got[b], want[b]) for b in range(batch)) <= 3 * bound      # a misplaced vector cannot hide in the norm


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("batch", [8, 16, 24, 32])
def test_sums_are_as_exact_as_the_tensor_memory_form(env, fmt, batch):
    """Against the exact product of the same fp16 operands (the weights as they come out for one-hot vectors).  16 mma in a row, each
    truncating at 2^-24 of a sum that grows to its end: 16 / 3 * 2^-24 = 3.2e-7 on average, twice that asked."""
    torch, F, ctx = env
    rows, cols = 200, 4096
    wt = torch.from_numpy(synth.host_tensor(fmt, rows, cols, seed=9)).cuda()
    ref = F.tensor_ref(wt.data_ptr(), 0, fmt, rows, cols)
    eye, w = torch.eye(cols, device="cuda"), torch.empty(cols, rows, device="cuda")
    for b in range(0, cols, 256):
        ctx.matvec(ref, eye[b:].data_ptr(), w[b:].data_ptr(), 256, cols, rows)
    x, y = torch.from_numpy(synth.host_x(cols, batch, seed=batch)).cuda(), torch.full((batch, rows), float("nan"), device="cuda")
    ctx.matvec(ref, x.data_ptr(), y.data_ptr(), batch, cols, rows)
    torch.cuda.synchronize()
    want = x.half().double() @ w.double()
    assert float((y.double() - want).norm() / want.norm()) <= 6.4e-7


def test_a_captured_product_repeats_its_bits(env):
    torch, F, _ = env
    rows, cols = 256, 1024
    ctx = F.Context(0)
    w, x = synth.host_tensor(synth.Q4_K, rows, cols, seed=1), synth.host_x(cols, 32, seed=2)
    wt, xt, y = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda(), torch.zeros(32, rows, device="cuda")
    ref = F.tensor_ref(wt.data_ptr(), 0, synth.Q4_K, rows, cols)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ctx.matvec(ref, xt.data_ptr(), y.data_ptr(), 32, cols, rows, side.cuda_stream)
    torch.cuda.synchronize()
    want = y.clone()
    y.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ctx.matvec(ref, xt.data_ptr(), y.data_ptr(), 32, cols, rows, torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert ctx.status() == 0
    del graph
    ctx.close()
