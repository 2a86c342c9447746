"""Shared-weight 'uvw': the FP64 GEMM kernels and the joined products of the FP32 backward pass at remainders of their
tiles (64 channels, 64 row-component pairs, 32 deep), one row, several shares of the rows, and paths that do not all fit
one joined block."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from helpers import REL_TOL, rel_err, tp_inputs, to_e3nn, to_oeq

pytestmark = pytest.mark.gpu

CASES = [
    ("64x0e+64x1o+64x2e", "0e+1o+2e", "64x0e+64x1o+64x2e", 1),
    ("64x0e+64x1o+64x2e", "0e+1o+2e", "64x0e+64x1o+64x2e", 300),
    ("64x0e+64x1o+64x2e", "0e+1o+2e", "64x0e+64x1o+64x2e", 1900),  # too many rows to deal the outputs over CTAs
    ("16x0e+80x1o", "0e+1o", "65x0e+16x1o+33x2e", 63),          # (33 and 65: not on the tensor cores)
    ("48x1o+16x3o", "1o+2e", "16x0e+64x2e+32x4e", 130),
    ("128x0e+128x1o", "0e+1o+2e", "128x0e+128x1o", 70),          # joined blocks of one path each
    ("16x0e+16x1o", "0e+1o", "16x0e+16x1o+16x4e", 40),           # an output irrep without paths
]


@pytest.mark.parametrize("in1,in2,out,batch", CASES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_shared_weights(in1, in2, out, batch, dtype):
    p = oeq.FullyConnectedTPProblem(in1, in2, out, irrep_dtype=dtype, weight_dtype=dtype)
    x, y, w, dz = tp_inputs(p, batch, 17)
    w = (w / 8).astype(dtype)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    tp = oeq.TensorProduct(p, torch_op=True)
    got = [tp(*dev[:3]), *tp.backward_helper(*dev)]
    again = tp.backward_helper(*dev)
    tp.check_device_status()
    assert all(torch.equal(a, b) for a, b in zip(got[1:], again))
    if dtype is np.float64:     # (the GEMM kernels are those that ran: two buffers of two 32 x 66 tiles)
        assert [tp.internal.launch_info(which)["smem_bytes"] for which in (0, 1)] == [4 * 32 * 66 * 8] * 2
        assert tp.internal.launch_info(1)["registers"] > 0
    want = [orc.tp_forward(p, x, y, w), *orc.tp_backward(p, x, y, w, dz)]
    for g, r in zip(got[:3], want):
        assert rel_err(g.cpu().numpy(), r) < REL_TOL[dtype]
    assert rel_err(to_e3nn(p, got[3].cpu().numpy()), want[3]) < REL_TOL[dtype]


def test_fp64_workspace_off_the_16_byte_rule():
    """A workspace at an odd multiple of 8 bytes is taken: the tiled kernel."""
    p = oeq.FullyConnectedTPProblem("16x0e+16x1o", "0e+1o", "16x0e+16x1o", irrep_dtype=np.float64, weight_dtype=np.float64)
    x, y, w, dz = tp_inputs(p, 50, 17)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    handle = oeq.TensorProduct(p).internal
    size = handle.workspace_bytes(50)
    got = [torch.empty_like(t) for t in dev[:3]]
    ws = torch.empty(size + 8, dtype=torch.uint8, device="cuda")
    handle.backward(50, *(t.data_ptr() for t in (*dev, *got)), ws.data_ptr() + 8, size, torch.cuda.current_stream().cuda_stream)
    want = orc.tp_backward(p, x, y, w, dz)
    for g, r in zip((got[0].cpu().numpy(), got[1].cpu().numpy(), to_e3nn(p, got[2].cpu().numpy())), want):
        assert rel_err(g, r) < REL_TOL[np.float64]


# one path or few products a row: small batches (and some large ones) are for the tiled kernel; both sides of each line
@pytest.mark.parametrize("irreps", [("16x0e", "0e", "16x0e"), ("32x0e", "0e", "32x0e"), ("128x0e", "0e", "64x0e"),
                                    ("16x0e+16x1o", "0e+1o", "16x0e+16x1o"), ("20x0e+20x1o+20x2e", "0e+1o+2e", "20x0e+20x1o+20x2e")],
                         ids=["16", "32", "128_64", "16_l1", "20_l2"])
@pytest.mark.parametrize("batch", [127, 128, 2368, 2369, 29601])
def test_fp64_lines_between_the_kernels(irreps, batch):
    p = oeq.FullyConnectedTPProblem(*irreps, irrep_dtype=np.float64, weight_dtype=np.float64)
    x, y, w, dz = tp_inputs(p, batch, 23)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    tp = oeq.TensorProduct(p, torch_op=True)
    got = [tp(*dev[:3]), *tp.backward_helper(*dev)]
    tp.check_device_status()
    some = np.r_[0:3, batch // 2, batch - 3:batch]                 # (the oracle is slow)
    want = [orc.tp_forward(p, x[some], y[some], w), *orc.tp_backward(p, x[some], y[some], w, dz[some])[:2]]
    for g, r in zip(got[:3], want):
        assert rel_err(g.cpu().numpy()[some], r) < REL_TOL[np.float64]
    parts = sum(orc.tp_backward(p, x[i:i + 5000], y[i:i + 5000], w, dz[i:i + 5000])[2] for i in range(0, batch, 5000))
    assert rel_err(to_e3nn(p, got[3].cpu().numpy()), parts) < REL_TOL[np.float64]
