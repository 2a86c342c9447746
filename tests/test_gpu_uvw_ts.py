"""Shared-weight FP32 'uvw' with a batch row per lane (forward with the weights in tensor memory, unless the problem has too few slices
of 32 input channels for it; weight gradient): one row to several tiles of 16 or 8 rows per CTA, fewer CTAs than outputs, multiplicities that are no multiple of 32 (padded slices) and
narrower than 64 (padded weight rows), a component count of seven, second inputs too long for registers, arrays off a 16-byte
boundary, an output without paths."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from helpers import rel_err, tp_inputs, to_e3nn, to_oeq

pytestmark = pytest.mark.gpu

SHAPES = {"even": ("64x0e+64x1o+64x2e", "0e+1o+2e", "64x0e+64x1o+64x2e"),
          "padded": ("36x0e+20x1o", "0e+1o+2e", "16x0e+48x1o+32x2e+16x4e"),     # (4e: no paths)
          "seven": ("8x2e+32x3o", "0e+1o", "16x3o+16x2e"),
          "long_y": ("32x0e+4x1o", "0e+1o+2e+3o+4e", "16x0e+16x1o+16x2e"),
          # the same features in problems whose forward pass has the weights in tensor memory
          "padded_ts": ("36x1o+20x2e", "0e+1o+2e", "16x0e+48x1o+32x2e+16x5o"),              # (5o: no paths)
          "seven_ts": ("8x2e+32x3o+32x1o", "0e+1o+2e", "16x3o+16x2e+32x1o"),
          "long_y_ts": ("32x2e+4x3o", "0e+1o+2e+3o+4e", "16x0e+16x1o+16x2e"),
          "mixed": ("64x0e+64x1o+64x2e+32x0o", "0e+1o+2e", "64x1o+64x2e+16x0o")}          # eight slices and one
STAGES = {shape: 4 if shape in ("even", "mixed") or shape.endswith("_ts") else 2 for shape in SHAPES}   # four: weights in tensor memory


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("rows", [1, 15, 16, 17, 33, 5003])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward(shape, rows, offset):
    p = oeq.FullyConnectedTPProblem(*SHAPES[shape])
    tp = oeq.TensorProduct(p, torch_op=True)
    assert tp.internal.launch_info(0)["stages"] == STAGES[shape]
    x, y, w, _ = tp_inputs(p, rows, 7)
    w = (w / np.sqrt(max(1, p.weight_numel / len(p.instructions)))).astype(np.float32)

    def device(a):
        flat = torch.from_numpy(np.ascontiguousarray(a)).cuda().flatten()
        return torch.cat((flat.new_zeros(offset), flat))[offset:].view(a.shape)

    xt, yt, wt = device(x), device(y), device(to_oeq(p, w))
    z = tp(xt, yt, wt)
    torch.cuda.synchronize()
    tp.check_device_status()
    # sums of up to 256 products in FP32, hi and lo parts of 11 bits each: 2^-22 per product, and T's rounding
    assert rel_err(z.cpu().numpy(), orc.tp_forward(p, x, y, w)) < 5e-6
    for n in (1, rows // 2):            # a row's sums do not depend on the batch that it is part of
        assert torch.equal(z[:n], tp(xt[:n].contiguous(), yt[:n].contiguous(), wt))


def test_rows_off_a_boundary():
    """Output rows that start off a 16-byte boundary."""
    p = oeq.FullyConnectedTPProblem(*SHAPES["even"])
    tp = oeq.TensorProduct(p, torch_op=True)
    x, y, w, _ = tp_inputs(p, 40, 9)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w))]
    want = tp(*dev)
    out = torch.zeros(want.numel() + 1, device="cuda")
    tp.internal.forward(40, *(t.data_ptr() for t in dev), out.data_ptr() + 4, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(out[1:].view_as(want), want) and out[0] == 0


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("rows", [1, 7, 8, 9, 25, 5003])
@pytest.mark.parametrize("shape", SHAPES)
def test_weight_gradient(shape, rows, offset):
    """Weight gradient from tiles of eight rows: fewer than a tile, remainders, several tiles per CTA and slot of the ring."""
    p = oeq.FullyConnectedTPProblem(*SHAPES[shape])
    tp = oeq.TensorProduct(p, torch_op=True)
    x, y, w, dz = tp_inputs(p, rows, 11)

    def device(a):
        flat = torch.from_numpy(np.ascontiguousarray(a)).cuda().flatten()
        return torch.cat((flat.new_zeros(offset), flat))[offset:].view(a.shape)

    args = [device(a) for a in (x, y, to_oeq(p, w), dz)]
    dw = tp.backward_helper(*args)[2]
    torch.cuda.synchronize()
    tp.check_device_status()
    # sums over rows and components in FP32 (their order differs from CTA to CTA), products as above
    assert rel_err(to_e3nn(p, dw.cpu().numpy()), orc.tp_backward(p, x, y, w, dz)[2]) < 5e-6
    for _ in range(3):
        assert torch.equal(tp.backward_helper(*args)[2], dw)


# On both sides of the rows up to which the wider kernel deals its groups of paths (148 SMs; five and six groups), and from which it has the
# weight gradients of scalar outputs.
@pytest.mark.parametrize("irreps,rows", [(SHAPES["even"], 768), (SHAPES["even"], 769), (SHAPES["mixed"], 928), (SHAPES["mixed"], 929),
                                         (("64x0e", "0e", "16x0e"), 14_800), (("64x0e", "0e", "16x0e"), 14_801)])
def test_weight_gradient_kernels_by_rows(irreps, rows):
    p = oeq.FullyConnectedTPProblem(*irreps)
    tp = oeq.TensorProduct(p, torch_op=True)
    x, y, w, dz = tp_inputs(p, rows, 17)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    dw = tp.backward_helper(*args)[2]
    tp.check_device_status()
    assert rel_err(to_e3nn(p, dw.cpu().numpy()), orc.tp_backward(p, x, y, w, dz)[2]) < 5e-6         # (as in test_weight_gradient)
    assert torch.equal(tp.backward_helper(*args)[2], dw)


def test_weight_gradient_of_many_rows():
    """The chains of additions within an accumulator have a length that does not grow with the batch."""
    p = oeq.FullyConnectedTPProblem("64x2e", "0e", "64x2e")
    tp = oeq.TensorProduct(p, torch_op=True)
    rows, want = 600_000, 0
    gen = torch.Generator(device="cuda").manual_seed(5)
    x, y, w, dz = (torch.randn(*s, device="cuda", generator=gen)
                   for s in ((rows, p.irreps_in1.dim), (rows, 1), (p.weight_numel,), (rows, p.irreps_out.dim)))
    dw = to_e3nn(p, tp.backward_helper(x, y, w, dz)[2].cpu().numpy())
    tp.check_device_status()
    for part in range(0, rows, 50_000):
        s = slice(part, part + 50_000)
        want = want + torch.einsum("buk,bwk->uw", (x[s].double() * y[s].double()).unflatten(1, (64, 5)), dz[s].double().unflatten(1, (64, 5)))
    want = want.flatten().cpu().numpy() * p.instructions[0].path_weight / np.sqrt(5)        # (the coefficients of 2e x 0e are 1 / sqrt(5))
    # 320 additions a chain, each off by at most 2^-23 of the sum so far, against 2 500 in a CTA's share of the rows (9e-5 measured)
    assert rel_err(dw, want) < 320 * 2 ** -23


@pytest.mark.parametrize("rows", [20, 100, 1000])
@pytest.mark.parametrize("irreps", [SHAPES["even"], SHAPES["seven"], ("64x0e", "0e", "64x0e")], ids=["even", "seven", "one"])
def test_weight_gradient_in_the_least_workspace(irreps, rows):
    """The order of the sums does not depend on how many partial weight gradients the workspace holds."""
    p = oeq.FullyConnectedTPProblem(*irreps)
    tp = oeq.TensorProduct(p)
    x, y, w, dz = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in tp_inputs(p, rows, 19))
    grads = [torch.empty_like(t) for t in (x, y, w)]
    stream, stated = torch.cuda.current_stream().cuda_stream, tp.internal.workspace_bytes(rows)
    ws = torch.empty(stated, dtype=torch.uint8, device="cuda")

    def gradient(size):
        tp.internal.backward(rows, *(t.data_ptr() for t in (x, y, w, dz, *grads, ws)), size, stream)
        return grads[2].clone()

    want, part = gradient(stated), p.weight_numel * 4
    accepted = []
    for n in range(1, stated // part):
        try:
            got = gradient(n * part)
        except RuntimeError as e:
            assert "workspace too small" in str(e) and not accepted
            continue
        assert torch.equal(got, want)
        accepted.append(n)
        if len(accepted) == 3:
            break
    assert accepted and accepted[0] <= (rows + 3) // 4


@pytest.mark.parametrize("few", [32, 64, 96])
def test_fewer_slices_than_producer_sets(few, monkeypatch):
    """An output of one to three slices of input channels: producer sets without a slice in a tile read its inputs too.  Hundreds
    of tiles per CTA, so that input buffers are filled again and again; every row against the FMA kernel."""
    p = oeq.FullyConnectedTPProblem(f"64x0e+64x1o+64x2e+{few}x0o", "0e+1o+2e", "64x1o+64x2e+16x0o")
    rows = 150_007
    gen = torch.Generator(device="cuda").manual_seed(3)
    x, y, w = (torch.randn(*s, device="cuda", generator=gen) for s in ((rows, p.irreps_in1.dim), (rows, p.irreps_in2.dim), (p.weight_numel,)))
    tp = oeq.TensorProduct(p, torch_op=True)
    assert tp.internal.launch_info(0)["stages"] == 4
    z = tp(x, y, w)
    tp.check_device_status()
    monkeypatch.setenv("OEQ_B200_UVW_TC", "0")
    want = oeq.TensorProduct(p, torch_op=True)(x, y, w)
    for o in p.irreps_out.slices():
        assert ((z[:, o] - want[:, o]).abs().max() / want[:, o].abs().max()).item() < 1e-5          # (5e-6 each, as in test_forward)


def test_gradients_of_many_outputs():
    """The barriers of the row-per-lane weight gradient beside its operands fit for 23 output irreps; more are for the wider kernel,
    with the shared memory of its own."""
    p = oeq.FullyConnectedTPProblem("16x0e", "0e", " + ".join(["16x0e"] * 24))
    tp = oeq.TensorProduct(p, torch_op=True)
    x, y, w, dz = tp_inputs(p, 500, 13)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)]
    dx, dy, dw = tp.backward_helper(*args)
    tp.check_device_status()
    for got, want in zip((dx.cpu().numpy(), dy.cpu().numpy(), to_e3nn(p, dw.cpu().numpy())), orc.tp_backward(p, x, y, w, dz)):
        assert rel_err(got, want) < 5e-6
