"""The steps either side of a product, fused into it (orome_cuda_fuse_next): the residual add + sum of squares as
the epilogue of the producing product (shaders.metal:86-124) and the RMS norm as the prologue of the products that
read the normalised vector (shaders.metal:126-149), as engine.m:625-653 strings them together.  Checked against the
numpy restatement of the two shader kernels in oracle/ and the fp64 matvec oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle
from orome_b200 import synth

pytestmark = pytest.mark.gpu

REL_L2_TOL = 1e-4
EPS = 1e-6


def rel_l2(got, want):
    want = np.asarray(want, np.float64)
    return float(np.linalg.norm(np.asarray(got, np.float64) - want) / max(np.linalg.norm(want), 1e-300))


@pytest.fixture(scope="module")
def env():
    import torch
    from orome_b200 import format as F
    ctx = F.Context(0)
    yield torch, F, ctx
    assert ctx.status() == 0
    ctx.close()


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def bf16_weights(n, seed):
    w = (1.0 + 0.25 * np.random.default_rng(seed).standard_normal(n)).astype(np.float32)
    return (w.view(np.uint32) >> 16).astype(np.uint16)


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("variant", [0, 1])
def test_output_projection_then_ffn_with_the_norm_in_between(env, fmt, variant):
    torch, F, ctx = env
    if variant == 1 and fmt in (synth.Q8_0, synth.Q6_K):
        pytest.skip("one scale layout")
    H, M = 2048, 1536
    wo, wg, wu = (synth.host_tensor(fmt, r, H, seed=s) for r, s in ((H, 11), (M, 12), (M, 13)))
    attn, resid = synth.host_x(H, seed=14), synth.host_x(H, seed=15)
    resid[7], resid[100] = 7e4, -9e4                                   # beyond the clamp
    nw = bf16_weights(H, 16)
    t = {k: dev(torch, v) for k, v in dict(wo=wo, wg=wg, wu=wu, attn=attn, resid=resid, nw=nw).items()}
    parts = torch.full((F.SUM_SQ_PARTS,), float("nan"), device="cuda")
    hidden = torch.full((H,), float("nan"), device="cuda")
    act = torch.full((M,), float("nan"), device="cuda")
    ref = lambda w, rows: F.tensor_ref(w.data_ptr(), 0, fmt, rows, H, variant)

    # 1. hidden = clamp(resid + Wo attn), partial sums of hidden^2
    ctx.fuse_next(None, F.ResidualEpilogue(t["resid"].data_ptr(), parts.data_ptr()))
    ctx.matvec(ref(t["wo"], H), t["attn"].data_ptr(), hidden.data_ptr())
    torch.cuda.synchronize()
    prod = oracle.matvec_f64(fmt, wo, H, H, attn, layout=variant)
    want_hidden, want_parts = oracle.residual_add_sum_sq(resid, prod.astype(np.float32))
    got_hidden, got_parts = hidden.cpu().numpy(), parts.cpu().numpy()
    assert got_hidden[7] == np.float32(65504.0) and got_hidden[100] == np.float32(-65504.0)
    assert rel_l2(got_hidden, want_hidden) <= REL_L2_TOL
    assert np.isfinite(got_parts).all() and (got_parts >= 0).all() and np.count_nonzero(got_parts) <= 296
    assert abs(float(got_parts.astype(np.float64).sum()) / float(want_parts.astype(np.float64).sum()) - 1.0) <= 1e-5

    # 2. act = silu(Wg n) * (Wu n) with n = hidden * rsqrt(sum / H + eps) * w read on the fly
    ctx.fuse_next(F.NormPrologue(t["nw"].data_ptr(), parts.data_ptr(), EPS), None)
    ctx.gate_up_swiglu(ref(t["wg"], M), ref(t["wu"], M), hidden.data_ptr(), act.data_ptr())
    torch.cuda.synchronize()
    n = oracle.rms_norm_apply_partial(got_hidden, nw, want_parts, EPS)
    want_act = oracle.swiglu_f64(oracle.matvec_f64(fmt, wg, M, H, n, layout=variant), oracle.matvec_f64(fmt, wu, M, H, n, layout=variant))
    assert rel_l2(act.cpu().numpy(), want_act) <= REL_L2_TOL

    # 3. the same prologue on a group of tensors (q / k / v read the normalised vector too), residual added in place
    q, k = torch.full((M,), float("nan"), device="cuda"), torch.full((M,), float("nan"), device="cuda")
    ctx.fuse_next(F.NormPrologue(t["nw"].data_ptr(), parts.data_ptr(), EPS))
    ctx.matvec_group([ref(t["wg"], M), ref(t["wu"], M)], hidden.data_ptr(), [q.data_ptr(), k.data_ptr()])
    torch.cuda.synchronize()
    assert rel_l2(q.cpu().numpy(), oracle.matvec_f64(fmt, wg, M, H, n, layout=variant)) <= REL_L2_TOL
    assert rel_l2(k.cpu().numpy(), oracle.matvec_f64(fmt, wu, M, H, n, layout=variant)) <= REL_L2_TOL
    inplace = t["resid"].clone()
    ctx.fuse_next(None, F.ResidualEpilogue(inplace.data_ptr(), parts.data_ptr()))
    ctx.matvec(ref(t["wo"], H), t["attn"].data_ptr(), inplace.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(inplace.cpu().numpy(), got_hidden)
    # a plain launch afterwards is a plain launch: the request does not linger
    plain = torch.empty((H,), device="cuda")
    ctx.matvec(ref(t["wo"], H), t["attn"].data_ptr(), plain.data_ptr())
    torch.cuda.synchronize()
    assert rel_l2(plain.cpu().numpy(), prod) <= REL_L2_TOL


def test_prologue_and_epilogue_on_the_same_product(env):
    torch, F, ctx = env
    fmt, H = synth.Q8_0, 1024
    w = synth.host_tensor(fmt, H, H, seed=21)
    x, resid, nw = synth.host_x(H, seed=22), synth.host_x(H, seed=23), bf16_weights(H, 24)
    _, in_parts = oracle.residual_add_sum_sq(x, np.zeros(H, np.float32))
    pin = np.zeros(F.SUM_SQ_PARTS, np.float32)
    pin[:in_parts.size] = in_parts                                     # a caller may fill the array itself
    t = {k: dev(torch, v) for k, v in dict(w=w, x=x, resid=resid, nw=nw, pin=pin).items()}
    pout = torch.full((F.SUM_SQ_PARTS,), float("nan"), device="cuda")
    y = torch.empty((H,), device="cuda")
    ctx.fuse_next(F.NormPrologue(t["nw"].data_ptr(), t["pin"].data_ptr(), EPS), F.ResidualEpilogue(t["resid"].data_ptr(), pout.data_ptr()))
    ctx.matvec(F.tensor_ref(t["w"].data_ptr(), 0, fmt, H, H), t["x"].data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    n = oracle.rms_norm_apply_partial(x, nw, in_parts, EPS)
    want, want_parts = oracle.residual_add_sum_sq(resid, oracle.matvec_f64(fmt, w, H, H, n).astype(np.float32))
    assert rel_l2(y.cpu().numpy(), want) <= REL_L2_TOL
    assert abs(float(pout.cpu().numpy().astype(np.float64).sum()) / float(want_parts.astype(np.float64).sum()) - 1.0) <= 1e-5


def test_calls_without_a_fused_form_drop_the_request(env):
    torch, F, ctx = env
    fmt, H = synth.Q8_0, 512
    w = dev(torch, synth.host_tensor(fmt, H, H, seed=31))
    x8, y8 = dev(torch, synth.host_x(H, 8, seed=32)), torch.zeros((8, H), device="cuda")
    nw, parts = dev(torch, bf16_weights(H, 33)), torch.zeros((F.SUM_SQ_PARTS,), device="cuda")
    ref = F.tensor_ref(w.data_ptr(), 0, fmt, H, H)
    pro = F.NormPrologue(nw.data_ptr(), parts.data_ptr(), EPS)
    epi = F.ResidualEpilogue(x8.data_ptr(), parts.data_ptr())
    ctx.fuse_next(pro)
    with pytest.raises(F.OromeError) as e:
        ctx.matvec(ref, x8.data_ptr(), y8.data_ptr(), 8, H, H)                   # batched
    assert e.value.code == F.ENOTSUP
    ctx.fuse_next(None, epi)
    with pytest.raises(F.OromeError) as e:
        ctx.gate_up_swiglu(ref, ref, x8.data_ptr(), y8.data_ptr())               # no residual form of the fused gate/up
    assert e.value.code == F.ENOTSUP
    ctx.fuse_next(None, epi)
    with pytest.raises(F.OromeError) as e:
        ctx.matvec_group([ref, ref], x8.data_ptr(), [y8[0].data_ptr(), y8[1].data_ptr()])     # epilogue wants one tensor
    assert e.value.code == F.ENOTSUP
    ctx.chain_begin()
    ctx.fuse_next(pro)
    with pytest.raises(F.OromeError) as e:
        ctx.matvec(ref, x8.data_ptr(), y8.data_ptr())                            # recordings have no fused form
    assert e.value.code == F.ENOTSUP
    ctx.matvec(ref, x8.data_ptr(), y8.data_ptr())
    ctx.chain_end().close()
    with pytest.raises(F.OromeError) as e:
        ctx.fuse_next(F.NormPrologue(nw.data_ptr() + 2, parts.data_ptr(), EPS))  # misaligned weights
    assert e.value.code == F.EINVAL
    y = torch.empty((H,), device="cuda")
    ctx.matvec(ref, x8.data_ptr(), y.data_ptr())                                 # nothing is pending any more
    torch.cuda.synchronize()
    want = oracle.matvec_f64(fmt, synth.host_tensor(fmt, H, H, seed=31), H, H, synth.host_x(H, 8, seed=32)[0])
    assert rel_l2(y.cpu().numpy(), want) <= REL_L2_TOL


@pytest.mark.parametrize("fmt", [synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("rows,cols", [(1, 256), (17, 512), (333, 2560), (2400, 4352), (48, 17408)])
@pytest.mark.parametrize("x_bits", [24, 16])
def test_fused_neighbours_on_both_kquant_kernels(env, fmt, rows, cols, x_bits):
    """Norm prologue and residual epilogue on one product at row-tile and superblock remainders, on the mma kernel and
    (OROME_OPT_KQUANT_MMA = 0) the dp4a kernel.  The mma kernel reads x as 32-bit fixed point at either option, so fp32 sums
    bound its error: a few 1e-7.  The dp4a kernel at 16 bits rounds x to 2^-16 of the largest of 32 elements, 1.9e-5 per
    element at a ratio of 2.1 between that and the deviation; a single row of 256 has a sum that may be small against
    its terms, hence the factor of ten."""
    torch, F, ctx = env
    w = synth.host_tensor(fmt, rows, cols, seed=31)
    x, resid, nw = synth.host_x(cols, seed=32), synth.host_x(rows, seed=33), bf16_weights(cols, 34)
    _, in_parts = oracle.residual_add_sum_sq(x, np.zeros(cols, np.float32))
    pin = np.zeros(F.SUM_SQ_PARTS, np.float32)
    pin[:in_parts.size] = in_parts
    t = {k: dev(torch, v) for k, v in dict(w=w, x=x, resid=resid, nw=nw, pin=pin).items()}
    n = oracle.rms_norm_apply_partial(x, nw, in_parts, EPS)
    prod = oracle.matvec_f64(fmt, w, rows, cols, n)
    err = []
    ctx.set_option(F.OPT_X_BITS, x_bits)
    try:
        for mma in (1, 0):
            ctx.set_option(F.OPT_KQUANT_MMA, mma)
            pout = torch.full((F.SUM_SQ_PARTS,), float("nan"), device="cuda")
            y = torch.full((rows,), float("nan"), device="cuda")
            ctx.fuse_next(F.NormPrologue(t["nw"].data_ptr(), t["pin"].data_ptr(), EPS), F.ResidualEpilogue(t["resid"].data_ptr(), pout.data_ptr()))
            ctx.matvec(F.tensor_ref(t["w"].data_ptr(), 0, fmt, rows, cols), t["x"].data_ptr(), y.data_ptr())
            torch.cuda.synchronize()
            got = y.cpu().numpy().astype(np.float64)
            err.append(rel_l2(got, np.clip(resid.astype(np.float64) + prod, -65504.0, 65504.0)))
            assert abs(float(pout.cpu().numpy().astype(np.float64).sum()) / float((got * got).sum()) - 1.0) <= 1e-5
    finally:
        ctx.set_option(F.OPT_KQUANT_MMA, 1)
        ctx.set_option(F.OPT_X_BITS, 24)
    print(f"fmt {fmt} {rows}x{cols} x_bits {x_bits}: mma {err[0]:.2e} dp4a {err[1]:.2e}")
    assert err[0] <= 2e-6
    assert err[1] <= (2e-6 if x_bits == 24 else 2e-4)


@pytest.mark.parametrize("rows,cols,stage_kb", [(5120, 17408, 0), (5120, 17408, 40), (4096, 17408, 20), (8192, 8192, 0), (3000, 5120, 0)])
def test_q6_ring_keeps_its_slots_apart(env, rows, cols, stage_kb):
    """Products back to back on rings of several stages a group, and on those whose shared memory would hold an odd number for two
    groups (three at 17408 columns with fused neighbours and 40-KiB stages, nine with 20-KiB ones; tests/test_mma_ring.py pins
    the plans): every repetition gives the first one's bits, and the first one is right."""
    torch, F, ctx = env
    fmt = synth.Q6_K
    w = synth.host_tensor(fmt, rows, cols, seed=41)
    x, resid = synth.host_x(cols, seed=42), synth.host_x(rows, seed=43)
    t = {k: dev(torch, v) for k, v in dict(w=w, x=x, resid=resid).items()}
    ref = F.tensor_ref(t["w"].data_ptr(), 0, fmt, rows, cols)
    out = torch.full((64, rows), float("nan"), device="cuda")
    parts = torch.zeros(F.SUM_SQ_PARTS, device="cuda")
    ctx.set_option(F.OPT_STAGE_KB, stage_kb)
    try:
        for i in range(64):
            if i % 2 == 0:
                ctx.fuse_next(None, F.ResidualEpilogue(t["resid"].data_ptr(), parts.data_ptr()))
            ctx.hint_next(ref)
            ctx.matvec(ref, t["x"].data_ptr(), out[i].data_ptr())
    finally:
        ctx.set_option(F.OPT_STAGE_KB, 0)
    torch.cuda.synchronize()
    assert ctx.status() == 0
    got = out.cpu().numpy()
    assert (got[0::2] == got[0]).all() and (got[1::2] == got[1]).all()
    pick = np.random.default_rng(44).choice(rows, 200, replace=False)
    rb = w.size // rows
    want = oracle.matvec_f64(fmt, np.ascontiguousarray(w.reshape(rows, rb)[pick]).reshape(-1), 200, cols, x)
    assert rel_l2(got[1][pick], want) <= 2e-6
    assert rel_l2(got[0][pick], np.clip(resid[pick].astype(np.float64) + want, -65504.0, 65504.0)) <= 2e-6
