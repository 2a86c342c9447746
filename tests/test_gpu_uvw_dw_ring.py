"""Weight gradient of shared-weight FP32 'uvw' products: the ring of operand stages has three slots from an output
multiplicity of 80 on and four below.  Enough rows that every CTA goes through the ring several times, two outputs so that
the ring goes on from one to the next; against the oracle, and repeatable."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from helpers import REL_TOL, rel_err, tp_inputs, to_e3nn, to_oeq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mul", [64, 80, 96, 128])
def test_ring_of_every_length(mul):
    p = oeq.FullyConnectedTPProblem(f"16x0e+{mul}x1o", "0e+1o", f"{mul}x0e+{mul}x1o")
    batch = 9973
    x, y, w, dz = tp_inputs(p, batch, 31)
    w = (w / 8).astype(np.float32)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    tp = oeq.TensorProduct(p, torch_op=True)
    dw = tp.backward_helper(*dev)[2]
    for _ in range(5):
        assert torch.equal(tp.backward_helper(*dev)[2], dw)
    tp.check_device_status()
    assert rel_err(to_e3nn(p, dw.cpu().numpy()), orc.tp_backward(p, x, y, w, dz)[2]) < REL_TOL[np.float32]
