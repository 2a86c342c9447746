"""Scratch memory of the deterministic convolution: a device that has none to spare; several streams, threads and graphs."""
import contextlib
import gc
import threading

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


def test_a_full_device_is_asked_once():
    """The size that did not fit is not tried again on every call (each try empties the allocator's cache)."""
    conv, (x, y, w, dz), index = _case(300_000)
    outputs = sum(-(-t.numel() * 4 // (2 * MB)) * 2 * MB for t in (x, y, w))
    with _memory_left(outputs + 8 * MB + int(0.3 * len(y) * conv.L1.dim * 4)):
        got = conv.backward_helper(x, y, w, dz, *index)
        failed = torch.cuda.memory_stats()["num_ooms"]
        for _ in range(3):
            got = None
            got = conv.backward_helper(x, y, w, dz, *index)
            assert conv.internal.last_backward_launches() == 9
        assert torch.cuda.memory_stats()["num_ooms"] == failed


# 300 000 edges: 346 MB, kept between calls; 100 000: from the allocator
@pytest.mark.parametrize("edges", [300_000, 100_000])
def test_two_streams(edges):
    """Backward passes of one operator on two streams at a time."""
    conv, first, index = _case(edges, seed=3)
    _, second, _ = _case(edges, seed=4)
    want = [[t.clone() for t in conv.backward_helper(*arrays, *index)] for arrays in (first, second)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(3):
        got = []
        for s, arrays in zip(streams, (first, second)):
            with torch.cuda.stream(s):
                got.append(conv.backward_helper(*arrays, *index))
        torch.cuda.synchronize()
        for g, r in zip(got, want):
            assert all(torch.equal(a, b) for a, b in zip(g, r))


def test_two_threads_on_one_stream():
    conv, first, index = _case(300_000, seed=3)
    _, second, _ = _case(300_000, seed=4)
    want = [[t.clone() for t in conv.backward_helper(*arrays, *index)] for arrays in (first, second)]
    same = [True, True]

    def run(i, arrays):
        for _ in range(10):
            got = conv.backward_helper(*arrays, *index)
            same[i] &= all(torch.equal(a, b) for a, b in zip(got, want[i]))

    threads = [threading.Thread(target=run, args=(i, a)) for i, a in enumerate((first, second))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert same == [True, True]


def test_a_captured_pass_has_scratch_of_its_own():
    """A graph that replays beside other calls of the operator."""
    conv, first, index = _case(300_000, seed=3)
    _, second, _ = _case(300_000, seed=4)
    want = [[t.clone() for t in conv.backward_helper(*arrays, *index)] for arrays in (first, second)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = conv.backward_helper(*first, *index)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        for t in captured:
            t.zero_()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            graph.replay()
        got = conv.backward_helper(*second, *index)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(captured, want[0]))
        assert all(torch.equal(a, b) for a, b in zip(got, want[1]))


def test_one_kept_buffer_for_all_entry_points():
    conv, (x, y, w, dz), index = _case(300_000)
    conv.backward_helper(x, y, w, dz, *index)
    held = torch.cuda.memory_allocated()
    conv._backward_impl(x, y, w, dz, *index)
    assert conv.workspace_size == len(y) * conv.L1.dim * 4
    address = conv.workspace_ptr
    conv._double_backward_impl(x, y, w, dz, x, y, w, *index)
    assert conv.workspace_ptr == address
    assert torch.cuda.memory_allocated() == held
