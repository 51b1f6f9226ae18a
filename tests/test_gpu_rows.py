"""Decoded rows are the oracle's bits wherever the output starts: 32-byte aligned (one store a piece) or only 16."""
import numpy as np
import pytest

import oracle
from orome_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K])
@pytest.mark.parametrize("rows,cols", [(1, 256), (3, 512), (37, 768), (130, 2048)])
@pytest.mark.parametrize("shift", [0, 4])
def test_rows_at_any_alignment(fmt, rows, cols, shift):
    import torch
    from orome_b200 import format as F
    ctx = F.Context(0)
    data = synth.host_tensor(fmt, rows, cols, seed=rows)
    w = torch.from_numpy(data).cuda()
    out = torch.full((rows * cols + 16,), float("nan"), device="cuda")
    ctx.dequant_rows(F.tensor_ref(w.data_ptr(), 0, fmt, rows, cols), 0, rows, out.data_ptr() + 4 * shift)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    want = oracle.decode_rows(fmt, data, rows, cols).reshape(-1)
    assert np.array_equal(got[shift:shift + rows * cols].view(np.uint32), want.view(np.uint32))
    assert np.isnan(got[:shift]).all() and np.isnan(got[shift + rows * cols:]).all()
    assert ctx.status() == 0
    ctx.close()
