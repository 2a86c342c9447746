"""The torch custom ops: schema, fake-tensor kernels and autograd registration (``torch.library.opcheck``), and
a ``torch.compile(fullgraph=True)`` call of each front end, as the reference's registration promises
(reference: openequivariance/implementations/TensorProductBase.py:236-298,
openequivariance/implementations/convolution/ConvolutionBase.py:560-709)."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from conftest import problem_by_name
from helpers import conv_inputs, random_graph, tp_inputs

pytestmark = pytest.mark.gpu

CHECKS = ("test_schema", "test_faketensor", "test_autograd_registration")


def _cuda(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


@pytest.mark.parametrize("name", ["nequip_32", "uvu_shared", "uvw_small"])
def test_tensor_product_ops(name):
    p = problem_by_name(name)
    tp = oeq.TensorProduct(p, torch_op=True)
    x, y, w, dz = tp_inputs(p, 9, 3)
    xt, yt, wt, dzt = _cuda(x, y, w, dz)
    torch.library.opcheck(tp.forward, (xt, yt, wt), test_utils=CHECKS)
    torch.library.opcheck(tp.backward_helper, (xt, yt, wt, dzt), test_utils=CHECKS)
    # fake tensors: shapes and dtypes without running a kernel
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode(allow_non_fake_inputs=False) as mode:
        fx, fy, fw = (mode.from_tensor(t) for t in (xt, yt, wt))
        fz = tp.forward(fx, fy, fw)
        assert tuple(fz.shape) == (9, p.irreps_out.dim) and fz.dtype == xt.dtype
    # compiled call: one graph, same numbers, gradients flow
    xg = xt.clone().requires_grad_(True)
    compiled = torch.compile(lambda a, b, c: tp.forward(a, b, c), fullgraph=True)
    z_c = compiled(xg, yt, wt)
    z_e = tp.forward(xt, yt, wt)
    assert torch.equal(z_c.detach(), z_e)
    z_c.backward(dzt)
    dx_e = tp.backward_helper(xt, yt, wt, dzt)[0]
    assert torch.equal(xg.grad, dx_e)


@pytest.mark.parametrize("deterministic", [False, True], ids=["atomic", "deterministic"])
def test_convolution_ops(deterministic):
    p = problem_by_name("nequip_32")
    nodes = 17
    rows, cols = random_graph(nodes, 90, seed=4)
    rows, cols, order, perm = orc.coord_graph(rows, cols)
    x, y, w, dz = conv_inputs(p, nodes, len(rows), 5)
    conv = oeq.TensorProductConv(p, torch_op=True, deterministic=deterministic)
    xt, yt, wt, dzt, r, c, pm = _cuda(x, y, w, dz, rows, cols, perm)
    index = (r, c, pm) if deterministic else (r, c)
    torch.library.opcheck(conv.forward, (xt, yt, wt, *index), test_utils=CHECKS)
    torch.library.opcheck(conv.backward_helper, (xt, yt, wt, dzt, *index), test_utils=CHECKS)
    xg = xt.clone().requires_grad_(True)
    compiled = torch.compile(lambda a, b, c_, *idx: conv.forward(a, b, c_, *idx), fullgraph=True)
    z_c = compiled(xg, yt, wt, *index)
    z_e = conv.forward(xt, yt, wt, *index)
    if deterministic:
        assert torch.equal(z_c.detach(), z_e)
    else:
        assert (z_c.detach() - z_e).abs().max().item() <= 1e-5 * z_e.abs().max().item()
    z_c.backward(dzt)
    dx_e = conv.backward_helper(xt, yt, wt, dzt, *index)[0]
    assert (xg.grad - dx_e).abs().max().item() <= 1e-5 * dx_e.abs().max().item()


@pytest.mark.parametrize("op", ["product", "convolution"])
def test_wrong_arguments_raise(op):
    """Messages name the shapes; the process lives on."""
    p = problem_by_name("nequip_32")
    rows, cols = random_graph(7, 40, seed=1)
    rows, cols, _, perm = orc.coord_graph(rows, cols)
    if op == "product":
        call, (x, y, w, dz), index = oeq.TensorProduct(p, torch_op=True), _cuda(*tp_inputs(p, 9, 1)), ()
    else:
        call = oeq.TensorProductConv(p, torch_op=True, deterministic=True)
        (x, y, w, dz), index = _cuda(*conv_inputs(p, 7, 40, 1)), _cuda(rows, cols, perm)
    for bad in ((x[:, 1:], y, w), (x, y[1:], w), (x, y, w[:, 1:]), (x.double(), y, w), (x, y, w.double())):
        with pytest.raises(ValueError, match=r"must be"):
            call.forward(*bad, *index)
    with pytest.raises(ValueError, match=r"output gradient must be \[\d+, 1120\]"):
        call.backward_helper(x, y, w, dz[:, 1:], *index)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        call.forward(x, y.cpu(), w, *index)
    if index:
        with pytest.raises(ValueError, match="int64"):
            call.forward(x, y, w, index[0].int(), *index[1:])
        with pytest.raises(ValueError, match="sender_perm"):
            call.forward(x, y, w, *index[:2], index[2][1:])
    assert torch.isfinite(call.forward(x, y, w, *index)).all()


@pytest.mark.parametrize("op", ["product", "convolution"])
def test_operands_whose_memory_does_not_hold_their_values(op):
    """Lazily negated operands and gradients give the gradients of their values; batched gradients are refused by name."""
    p = problem_by_name("nequip_32")
    rows, cols = random_graph(7, 40, seed=1)
    rows, cols, _, perm = orc.coord_graph(rows, cols)
    if op == "product":
        call, (x, y, w, dz), index = oeq.TensorProduct(p, torch_op=True), _cuda(*tp_inputs(p, 9, 1)), ()
    else:
        call = oeq.TensorProductConv(p, torch_op=True, deterministic=True)
        (x, y, w, dz), index = _cuda(*conv_inputs(p, 7, 40, 1)), _cuda(rows, cols, perm)

    gen = torch.Generator(device="cuda").manual_seed(2)
    cotangents = [torch.randn(t.shape, device="cuda", generator=gen) for t in (x, y, w)]

    def gradients(wrap_x, wrap_dz, second=False):
        ins = [t.clone().requires_grad_(True) for t in (x, y, w)]
        z = call.forward(wrap_x(ins[0]), *ins[1:], *index)
        if not second:
            return torch.autograd.grad(z, ins, wrap_dz(dz))
        first = torch.autograd.grad(z, ins, wrap_dz(dz), create_graph=True)
        return torch.autograd.grad(first, ins, (wrap_dz(cotangents[0]), *cotangents[1:]))

    negated, plain = torch._neg_view, torch.neg
    for second in (False, True):
        for wraps in ((negated, lambda t: t), (lambda t: t, negated), (negated, negated)):
            same = tuple(plain if f is negated else f for f in wraps)
            for got, want in zip(gradients(*wraps, second), gradients(*same, second)):
                assert (got - want).abs().max().item() <= 1e-5 * want.abs().max().item()
    z = call.forward(x.requires_grad_(True), y, w, *index)
    with pytest.raises(RuntimeError, match="Batching rule"):
        torch.autograd.grad(z, x, torch.stack([dz, dz]), is_grads_batched=True)


def test_first_calls_from_several_threads():
    """The kernels of an operator are loaded by its first call; several threads may make it."""
    import threading
    p = problem_by_name("nequip_32")
    rows, cols = random_graph(7, 40, seed=1)
    rows, cols, _, perm = orc.coord_graph(rows, cols)
    for _ in range(5):
        cases = [(oeq.TensorProduct(p, torch_op=True), _cuda(*tp_inputs(p, 9, 1)), ()),
                 (oeq.TensorProductConv(p, torch_op=True, deterministic=True), _cuda(*conv_inputs(p, 7, 40, 1)), _cuda(rows, cols, perm))]
        for op, (x, y, w, dz), index in cases:
            results, start = [None] * 6, threading.Barrier(6)

            def run(i):
                with torch.cuda.stream(torch.cuda.Stream()):
                    start.wait()
                    results[i] = [op.forward(x, y, w, *index), *op.backward_helper(x, y, w, dz, *index)]

            torch.cuda.synchronize()
            threads = [threading.Thread(target=run, args=(i,)) for i in range(6)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            torch.cuda.synchronize()
            want = [op.forward(x, y, w, *index), *op.backward_helper(x, y, w, dz, *index)]
            assert all(torch.equal(a, b) for got in results for a, b in zip(got, want))
