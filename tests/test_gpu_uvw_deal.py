"""Shared-weight FP32 'uvw' with the weights in shared memory (W dZ of every problem; the forward pass of some, two operand stages):
batches whose chunks of rows are dealt over the CTAs for all output irreps together.  A row's
sums do not depend on the CTA that forms them, so the rows of a dealt batch have the bits of the same rows in batches that
are too small to be dealt, and the latter are held against the oracle."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from helpers import REL_TOL, rel_err, tp_inputs, to_oeq

pytestmark = pytest.mark.gpu

PER_SM = 160        # rows per SM up to which a batch is dealt (more than 32 input channels; 200 below)


@pytest.mark.parametrize("rows", [1177, 1200, 4001, PER_SM * 148, PER_SM * 148 + 1, 200 * 148])
@pytest.mark.parametrize("irreps,stages", [(("64x0e+64x1o+64x2e", "0e+1o+2e", "64x0e+64x1o+64x2e"), 4),
                                           (("16x0e+48x1o", "0e+1o", "32x0e+16x1o+48x2e+16x4e"), 2),   # (4e: no paths)
                                           (("64x0e+64x1o", "0e+1o", "96x0e+16x1o+16x4e"), 2)],
                         ids=["even", "uneven", "wide"])
def test_dealt_rows(irreps, stages, rows):
    p = oeq.FullyConnectedTPProblem(*irreps)
    x, y, w, dz = tp_inputs(p, rows, 5)
    w = (w / 8).astype(np.float32)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    tp = oeq.TensorProduct(p, torch_op=True)
    assert tp.internal.launch_info(0)["stages"] == stages
    got = [tp(*dev[:3]), *tp.backward_helper(*dev)[:2]]
    blocks = [(0, 200), (rows // 2, rows // 2 + 300), (rows - 41, rows)]
    for lo, hi in blocks:
        part = [dev[0][lo:hi].contiguous(), dev[1][lo:hi].contiguous(), dev[2], dev[3][lo:hi].contiguous()]
        want = [tp(*part[:3]), *tp.backward_helper(*part)[:2]]
        assert all(torch.equal(g[lo:hi], r) for g, r in zip(got, want))
        ref = [orc.tp_forward(p, x[lo:hi], y[lo:hi], w), *orc.tp_backward(p, x[lo:hi], y[lo:hi], w, dz[lo:hi])[:2]]
        for g, r in zip(want, ref):
            assert rel_err(g.cpu().numpy(), r) < REL_TOL[np.float32]
    tp.check_device_status()
