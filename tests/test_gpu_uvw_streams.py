"""Shared-weight 'uvw' products of one operator on several streams at a time, each with weights of its own: what a call
prepares (weights in the operand layout of the tensor cores) belongs to the call."""
import gc

import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from helpers import tp_inputs, to_oeq

pytestmark = pytest.mark.gpu


# (with 0e: weights packed for the forward pass too, in FP32)
@pytest.mark.parametrize("in2", ["0e+1o", "0e"])
@pytest.mark.parametrize("entry", ["op", "python"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_overlapping_calls(dtype, entry, in2):
    p = oeq.FullyConnectedTPProblem("64x0e+64x1o", in2, "64x0e+64x1o", irrep_dtype=dtype, weight_dtype=dtype)
    tp = oeq.TensorProduct(p, torch_op=True)
    if dtype is np.float32:
        assert (tp.internal.forward_workspace_bytes() > 0) == (in2 == "0e")
    forward, backward = (tp.forward, tp.backward_helper) if entry == "op" else (tp._forward_impl, tp._backward_impl)
    inputs = []
    for seed in range(4):
        x, y, w, dz = tp_inputs(p, 3000, seed)
        inputs.append([torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz)])
    want = [[forward(*a[:3]), *backward(*a)] for a in inputs]
    streams = [torch.cuda.Stream() for _ in inputs]
    torch.cuda.synchronize()
    for _ in range(5):
        got = []
        for s, a in zip(streams, inputs):
            with torch.cuda.stream(s):
                got.append([forward(*a[:3]), *backward(*a)])
        torch.cuda.synchronize()
        for g, r in zip(got, want):
            assert all(torch.equal(a, b) for a, b in zip(g, r))


def test_less_workspace_than_stated():
    """The handle's own memory, blocks of the batch, or the tiled kernels take over; the results stay."""
    p = oeq.FullyConnectedTPProblem("64x0e+64x1o", "0e+1o", "64x0e+64x1o")
    tp = oeq.TensorProduct(p)
    batch = 20000
    x, y, w, dz = tp_inputs(p, batch, 5)
    x, y, w, dz = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y, to_oeq(p, w), dz))
    want = tp._backward_impl(x, y, w, dz)
    z = tp._forward_impl(x, y, w)
    stream, full = torch.cuda.current_stream().cuda_stream, tp.internal.workspace_bytes(batch)
    out = torch.empty_like(z)
    tp.internal.forward(batch, x.data_ptr(), y.data_ptr(), w.data_ptr(), out.data_ptr(), stream)
    assert torch.equal(out, z)
    for size in (full - 16, full // 4, 256 * p.weight_numel * 4):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        got = [torch.empty_like(t) for t in (x, y, w)]
        tp.internal.backward(batch, *(t.data_ptr() for t in (x, y, w, dz, *got, ws)), size, stream)
        for g, r in zip(got, want):
            assert (g - r).abs().max().item() <= 1e-5 * r.abs().max().item()


@pytest.mark.parametrize("entry", ["op", "python"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_a_full_device(dtype, entry):
    """The products of the weights with dZ (360 and 720 MB here) shrink to what there is."""
    p = oeq.FullyConnectedTPProblem("64x0e+64x1o", "0e+1o", "64x0e+64x1o", irrep_dtype=dtype, weight_dtype=dtype)
    tp = oeq.TensorProduct(p, torch_op=True)
    batch, mb = 100_000, 1 << 20
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, y, w, dz = (torch.randn(*s, device="cuda", dtype=torch.float32 if dtype is np.float32 else torch.float64, generator=gen)
                   for s in ((batch, p.irreps_in1.dim), (batch, p.irreps_in2.dim), (p.weight_numel,), (batch, p.irreps_out.dim)))
    call = tp.backward_helper if entry == "op" else tp._backward_impl
    want = call(x, y, w, dz)
    outputs = sum(-(-t.numel() * t.element_size() // (2 * mb)) * 2 * mb for t in (x, y)) + 22 * mb
    torch.cuda.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + outputs + 130 * mb) / total)
    try:
        got = call(x, y, w, dz)
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for g, r in zip(got, want):
        assert (g - r).abs().max().item() <= (1e-5 if dtype is np.float32 else 1e-12) * r.abs().max().item()
