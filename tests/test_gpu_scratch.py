"""Scratch memory of the deterministic convolution: a device that has none to spare."""
import contextlib
import gc

import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from conftest import problem_by_name
from helpers import random_graph

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _case(edges, nodes=5000, seed=3):
    p = problem_by_name("nequip_32")
    rows, cols = random_graph(nodes, edges, seed)
    rows, cols, _, perm = orc.coord_graph(rows, cols)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    arrays = [torch.randn(n, k, device="cuda", generator=gen) for n, k in ((nodes, p.irreps_in1.dim), (edges, p.irreps_in2.dim),
                                                                          (edges, p.weight_numel), (nodes, p.irreps_out.dim))]
    index = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rows, cols, perm)]
    return oeq.TensorProductConv(p, torch_op=True, deterministic=True), arrays, index


@contextlib.contextmanager
def _memory_left(spare):
    """At most `spare` bytes more than now from the caching allocator."""
    torch.cuda.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + spare) / total)
    try:
        yield
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


# scratch rows of 1 152 bytes: 230 MB and 346 MB.  A quarter of the former is too few rows to be of use (the sender-order
# kernel, one launch); of the latter it holds a quarter of the edges (four blocks of two launches and the clearing of dX).
@pytest.mark.parametrize("edges,share,launches", [(200_000, 1.0, 2), (200_000, 0.3, 1), (200_000, 0.0, 1),
                                                  (300_000, 1.0, 2), (300_000, 0.3, 9), (300_000, 0.0, 1)])
@pytest.mark.parametrize("entry", ["op", "python"])
def test_a_full_device(edges, share, launches, entry):
    conv, (x, y, w, dz), index = _case(edges)
    want = conv._backward_impl(x, y, w, dz, *index, scratch=False)
    row = conv.L1.dim * 4
    outputs = sum(-(-t.numel() * 4 // (2 * MB)) * 2 * MB for t in (x, y, w))
    call = conv.backward_helper if entry == "op" else conv._backward_impl
    with _memory_left(outputs + 8 * MB + int(share * edges * row)):
        got = call(x, y, w, dz, *index)
        assert conv.internal.last_backward_launches() == launches
    for g, r in zip(got, want):
        assert (g - r).abs().max().item() <= 1e-5 * r.abs().max().item()
