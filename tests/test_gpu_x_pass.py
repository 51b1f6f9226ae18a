"""The read of x at the head of a decode product: how its pieces are dealt out to warps, its alignment, its fixed-point scales.

Bound: 24-bit fixed point per group is good to 2^-24 of the group's largest element and its scale to 2^-24; with the fp32 sums
behind it a few 1e-7 of the result, 2e-6 asked (as elsewhere for 24-bit x)."""
import numpy as np
import pytest

import oracle
from orome_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    from orome_b200 import format as F
    ctx = F.Context(0)
    yield torch, F, ctx
    assert ctx.status() == 0
    ctx.close()


def _product(env, fmt, rows, cols, x, shift, nan=False):
    """matvec with x `shift` floats behind a 256-byte boundary: its relative error (nan: the product itself)."""
    torch, F, ctx = env
    w = synth.host_tensor(fmt, rows, cols, seed=cols + shift)
    wt = torch.from_numpy(w).cuda()
    buf = torch.zeros(cols + 64, device="cuda")
    buf[shift:shift + cols] = torch.from_numpy(x).cuda()
    y = torch.full((rows,), 0.0 if nan else float("nan"), device="cuda")
    ctx.matvec(F.tensor_ref(wt.data_ptr(), 0, fmt, rows, cols), buf.data_ptr() + 4 * shift, y.data_ptr())
    torch.cuda.synchronize()
    if nan:
        return y.cpu().numpy()
    want = oracle.matvec_f64(fmt, w, rows, cols, x)
    return float(np.linalg.norm(y.cpu().numpy() - want) / np.linalg.norm(want))


# one superblock; fewer and more superblocks than warps; one round of five a warp, and one superblock more than a round
@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("cols", [256, 2560, 5120, 17408, 19456, 20736])
@pytest.mark.parametrize("shift", [0, 4])      # 32- and 16-byte aligned
def test_widths_and_alignment(env, fmt, cols, shift):
    assert _product(env, fmt, 80, cols, synth.host_x(cols, seed=cols), shift) <= 2e-6


# groups of zeros beside others, and magnitudes at which a product of two scales leaves the range of fp32's normal numbers
@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("scale", [1e-25, 1.0, 1e25])
def test_scales_of_x(env, fmt, scale):
    x = synth.host_x(2048, seed=3)
    x[256:512] = 0.0
    x[512:768] *= 1e-6
    x[1024:1056] = 0.0
    assert _product(env, fmt, 48, 2048, (x * np.float32(scale)).astype(np.float32), 0) <= 2e-6


# an infinite element, and a group of nothing but NaN, are not lost among the zeros of the fixed point
@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_x_that_is_not_finite(env, fmt, bad):
    x = synth.host_x(1024, seed=4)
    x[256:512] = bad
    assert np.isnan(_product(env, fmt, 40, 1024, x, 0, nan=True)).all()


# norm and residual around one product; 21000 rows: more of them a CTA than its flush buffers (and the residuals read ahead) hold
@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("rows", [1, 40, 21000])
def test_norm_and_residual_around_a_product(env, fmt, rows):
    torch, F, ctx = env
    cols = 512
    w, x, res = synth.host_tensor(fmt, rows, cols, seed=5), synth.host_x(cols, seed=6), synth.host_x(rows, seed=7)
    nw = (synth.host_x(cols, seed=8).view(np.uint32) >> 16).astype(np.uint16)
    d = {k: torch.from_numpy(v).cuda() for k, v in dict(w=w, x=x, res=res, nw=nw.view(np.int16)).items()}
    parts, out = torch.zeros(F.SUM_SQ_PARTS, device="cuda"), torch.full((F.SUM_SQ_PARTS,), float("nan"), device="cuda")
    parts[:4] = float((x.astype(np.float64) ** 2).sum()) / 4
    y = torch.full((rows,), float("nan"), device="cuda")
    ctx.fuse_next(F.NormPrologue(d["nw"].data_ptr(), parts.data_ptr(), 1e-6), F.ResidualEpilogue(d["res"].data_ptr(), out.data_ptr()))
    ctx.matvec(F.tensor_ref(d["w"].data_ptr(), 0, fmt, rows, cols), d["x"].data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    xn = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean() + 1e-6) * (nw.astype(np.uint32) << 16).view(np.float32)
    want = res + oracle.matvec_f64(fmt, w, rows, cols, xn.astype(np.float32))
    got = y.cpu().numpy()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-6
    assert abs(float(out.double().sum()) / float((got.astype(np.float64) ** 2).sum()) - 1) <= 1e-5


# the same bound where x without 1 / rms would be out of the fixed point's range; zeros where its sum of squares is infinite
@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("bits,scale", [(24, 1e-31), (24, 1e-25), (24, 1e17), (24, 1e36), (16, 1e36)])
def test_magnitudes_of_a_normalised_x(env, fmt, bits, scale):
    torch, F, ctx = env
    rows, cols = 48, 2048
    w, nw = synth.host_tensor(fmt, rows, cols, seed=5), (synth.host_x(cols, seed=8).view(np.uint32) >> 16).astype(np.uint16)
    x = (synth.host_x(cols, seed=6) * np.float32(scale)).astype(np.float32)
    total = (x.astype(np.float64) ** 2).sum()
    wt, xt, nwt = (torch.from_numpy(a).cuda() for a in (w, x, nw.view(np.int16)))
    parts, y = torch.zeros(F.SUM_SQ_PARTS, device="cuda"), torch.full((rows,), float("nan"), device="cuda")
    parts[0] = total if total < 3e38 else float("inf")
    ctx.set_option(F.OPT_X_BITS, bits)
    try:
        ctx.fuse_next(F.NormPrologue(nwt.data_ptr(), parts.data_ptr(), 1e-6), None)
        ctx.matvec(F.tensor_ref(wt.data_ptr(), 0, fmt, rows, cols), xt.data_ptr(), y.data_ptr())
        torch.cuda.synchronize()
    finally:
        ctx.set_option(F.OPT_X_BITS, 24)
    got = y.cpu().numpy().astype(np.float64)
    if total > 3e38:
        assert (got == 0).all()
        return
    xn = x.astype(np.float64) / np.sqrt(total / cols + 1e-6) * (nw.astype(np.uint32) << 16).view(np.float32)
    want = oracle.decode_rows(fmt, w, rows, cols).reshape(rows, cols).astype(np.float64) @ xn
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-6
