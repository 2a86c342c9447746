"""'uvw' with per-row weights: the one-row-per-CTA kernels at chunk remainders of every multiplicity, second inputs of
multiplicity above one, one row, and more rows than CTAs; a problem whose row does not fit them, and large batches of rows
with few weights (tiled kernel)."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from helpers import REL_TOL, rel_err, tp_inputs, to_e3nn, to_oeq

pytestmark = pytest.mark.gpu

ODD = ("40x0e+9x1o+1x2e", "2x0e+3x1o", "36x0e+33x1o+5x1e+1x0o")
WIDE = ("128x2e+128x3o", "4x1o+4x2e", "16x2e+16x3o")


@pytest.mark.parametrize("irreps,batch", [(ODD, 1), (ODD, 7), (ODD, 2500), (WIDE, 3)], ids=["one", "few", "many", "tiled"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_row_weights(irreps, batch, dtype):
    p = oeq.FullyConnectedTPProblem(*irreps, shared_weights=False, irrep_dtype=dtype, weight_dtype=dtype)
    arrays = tp_inputs(p, batch, 3)
    x, y, w, dz = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*arrays[:2], to_oeq(p, arrays[2]), arrays[3]))
    tp = oeq.TensorProduct(p, torch_op=True)
    z = tp(x, y, w)
    dx, dy, dw = tp.backward_helper(x, y, w, dz)
    tp.check_device_status()
    if irreps is ODD:       # (the row kernels are those that ran: one row of each operand and of T in shared memory)
        size = sum(-(-n // 4) * 4 for n in (p.irreps_in1.dim, p.irreps_in2.dim, p.irreps_out.dim,
                                            sum(p.irreps_in1[i.i_in1].mul * p.irreps_in2[i.i_in2].mul * p.irreps_out[i.i_out].ir.dim
                                                for i in p.instructions)))
        assert tp.internal.launch_info(0)["smem_bytes"] == size * np.dtype(dtype).itemsize
    some = slice(0, batch) if batch < 100 else np.r_[0:3, batch // 2, batch - 3:batch]     # (the oracle is slow)
    sub = [a[some] for a in arrays]
    want = [orc.tp_forward(p, *sub[:3]), *orc.tp_backward(p, *sub)]
    for got, ref in zip((z, dx, dy), want):
        assert rel_err(got.cpu().numpy()[some], ref) < REL_TOL[dtype]
    assert rel_err(to_e3nn(p, dw.cpu().numpy()[some]), want[3]) < REL_TOL[dtype]


FEW = [("4x0e+4x1o", "0e+1o", "4x0e+4x1o"), ("8x0e+8x1o", "0e+1o", "8x0e+8x1o"), ("128x0e", "0e", "4x0e"), ("8x0e+8x1o+8x2e", "0e+1o+2e", "8x0e+8x1o+8x2e")]


# (on both sides of 8, 24 and 64 rows per SM, where batches of rows with few weights go over to the tiled kernel)
@pytest.mark.parametrize("batch", [1185, 3552, 3553, 9473])
@pytest.mark.parametrize("irreps", FEW, ids=["mul4", "mul8", "one_tile", "mul8_l2"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_few_weights(irreps, batch, dtype):
    test_row_weights(irreps, batch, dtype)


# Rows of whole 16-byte pieces: bulk copies of a row's arrays ahead of it.  Remainders of the chunks of 32 channels (33 ... 52)
# and of the units of 16, output channels beside which four, three, two and one input channels fit a warp, second inputs of
# multiplicity above one; more rows than two per CTA; arrays that start off a 16-byte boundary.
STAGED = [("40x0e+12x1o+4x2e", "1x0e+1x1o", "52x0e+8x1o+12x1e+4x0o"), ("36x0e+4x1o", "4x0e+4x1o", "16x0e+20x1o"),
          ("10x1o + 10x1e + 48x0e + 48x0o", "1x0e + 1x1o", "10x1o + 10x1e + 48x0e + 48x0o")]


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("batch", [1, 7, 1501])
@pytest.mark.parametrize("irreps", STAGED, ids=["tails", "mul_v", "docking"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_staged_rows(irreps, batch, offset, dtype):
    p = oeq.FullyConnectedTPProblem(*irreps, shared_weights=False, irrep_dtype=dtype, weight_dtype=dtype)
    assert all(n * np.dtype(dtype).itemsize % 16 == 0
               for n in (p.irreps_in1.dim, p.irreps_in2.dim, p.irreps_out.dim, p.weight_numel))
    arrays = tp_inputs(p, batch, 5)

    def device(a):
        flat = torch.from_numpy(np.ascontiguousarray(a)).cuda().flatten()
        return torch.cat((flat.new_zeros(offset), flat))[offset:].view(a.shape)

    x, y, w, dz = (device(a) for a in (*arrays[:2], to_oeq(p, arrays[2]), arrays[3]))
    tp = oeq.TensorProduct(p, torch_op=True)
    z = tp(x, y, w)
    dx, dy, dw = tp.backward_helper(x, y, w, dz)
    tp.check_device_status()
    some = slice(0, batch) if batch < 100 else np.r_[0:3, batch // 2, batch - 3:batch]
    sub = [a[some] for a in arrays]
    want = [orc.tp_forward(p, *sub[:3]), *orc.tp_backward(p, *sub)]
    for got, ref in zip((z, dx, dy), want):
        assert rel_err(got.cpu().numpy()[some], ref) < REL_TOL[dtype]
    assert rel_err(to_e3nn(p, dw.cpu().numpy()[some]), want[3]) < REL_TOL[dtype]
    # (a CTA has two rows' weights in shared memory; two such CTAs have to fit an SM, and those of 'docking' in FP64 do not)
    staged = [tp.internal.launch_info(which)["smem_bytes"] >= 2 * p.weight_numel * np.dtype(dtype).itemsize for which in (0, 1)]
    assert staged == [not (irreps is STAGED[2] and dtype is np.float64)] * 2
    again = (tp(x, y, w), *tp.backward_helper(x, y, w, dz))         # every row, not only those compared: the same bits
    for a, b in zip((z, dx, dy, dw), again):
        assert torch.equal(a, b)
