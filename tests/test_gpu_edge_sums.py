"""The edge sums of a shared-weight 'uvw' convolution (channel-wise, without weights): sums of products per receiver."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from openequivariance_b200.conv import UVWConvPlan, _UnitWeightConv
from openequivariance_b200.wigner import cg_nonzeros
from oracle import tp_oracle as orc
from helpers import REL_TOL, rel_err
from test_gpu_slice_conv import DEGREES, _unaligned

pytestmark = pytest.mark.gpu


def _edge_sum(mul, in1, in2, out, dtype=np.float32):
    wide = lambda irreps: "+".join(f"{mul}x{ir}" for ir in irreps.split("+"))
    return UVWConvPlan(oeq.FullyConnectedTPProblem(wide(in1), in2, wide(out), irrep_dtype=dtype, weight_dtype=dtype)).edge_sum


def _cuda(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _pairs(p):
    """[components of a channel of the first input, components of the second]: pairs with a coefficient."""
    d1 = np.cumsum([0] + [2 * ir.l + 1 for _, ir in p.irreps_in1])
    d2 = np.cumsum([0] + [2 * ir.l + 1 for _, ir in p.irreps_in2])
    has = np.zeros((d1[-1], d2[-1]), bool)
    for t in p.instructions:
        for i, j, _, _ in cg_nonzeros(p.irreps_in1[t.i_in1].ir.l, p.irreps_in2[t.i_in2].ir.l, p.irreps_out[t.i_out].ir.l):
            has[d1[t.i_in1] + i, d2[t.i_in2] + j] = True
    return has


def _components(p):
    """Component of its channel that each value of a first-input row is."""
    out, d = [], 0
    for mul, ir in p.irreps_in1:
        out.append(np.tile(d + np.arange(2 * ir.l + 1), mul))
        d += 2 * ir.l + 1
    return np.concatenate(out)


@pytest.mark.parametrize("deterministic", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("mul,dtype", [(64, np.float32), (32, np.float32), (8, np.float64)])
def test_infinite_components_stay_with_their_pairs(mul, dtype, deterministic):
    """An infinite component of one input reaches the gradients of the components that share a coefficient with it only."""
    p = _edge_sum(mul, "0e+1o+2e", "0e+1o+2e", "0e+1o+2e", dtype)
    has, comp = _pairs(p), _components(p)
    nodes, rng = 40, np.random.default_rng(5)
    rows, cols = np.arange(nodes), np.arange(nodes)[::-1].copy()        # one edge per receiver and per sender
    x, y, dz = (rng.normal(size=(nodes, r.dim)).astype(dtype) for r in (p.irreps_in1, p.irreps_in2, p.irreps_out))
    ones = np.ones((nodes, p.weight_numel), dtype)
    conv = _UnitWeightConv(p, deterministic)
    index = _cuda(rows, cols) + (_cuda(cols) if deterministic else [])
    assert not has.all()
    i0, j0 = np.argwhere(~has)[0]
    for where, kept_x, kept_y in (("y", ~has[:, j0][comp], np.arange(has.shape[1]) != j0),
                                  ("x", comp != i0, ~has[i0])):
        hot, zeroed = {"x": x.copy(), "y": y.copy()}, {"x": x.copy(), "y": y.copy()}
        at = (slice(None), comp == i0) if where == "x" else (slice(None), j0)
        hot[where][at], zeroed[where][at] = np.inf, 0
        dx, dy = conv.backward_helper(*_cuda(hot["x"], hot["y"], dz), *index)
        rx, ry, _ = orc.conv_backward(p, zeroed["x"], zeroed["y"], ones, dz, rows, cols)
        assert rel_err(dx.cpu().numpy()[:, kept_x], rx[:, kept_x]) < REL_TOL[dtype]
        assert rel_err(dy.cpu().numpy()[:, kept_y], ry[:, kept_y]) < REL_TOL[dtype]


# Both sides of the lines between the forms: per edge or sums of products, one or two channels per lane, rows of at most 32
# channels, one slice and several; FP64 with and without sums in the backward pass.
E1, E2, E3 = "0e+1o", "0e+1o+2e", "0e+1o+2e+3o"
WALKS = [(8, E1, E1, E1, np.float32), (20, E2, E2, E2, np.float32), (32, E1, E1, E2, np.float32), (64, E2, E2, "0e", np.float32),
         (64, E3, E2, E3, np.float32), (96, E2, E2, E2, np.float32), (128, E2, E2, E2, np.float32), (256, E2, E2, E2, np.float32),
         (8, E1, E1, E1, np.float64), (24, E2, E2, E2, np.float64), (64, E1, E1, E1, np.float64), (128, E1, E2, E1, np.float64)]


@pytest.mark.parametrize("deterministic", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("graph", ["one_edge", "runs", "many"])
@pytest.mark.parametrize("mul,in1,in2,out,dtype", WALKS)
def test_walk(mul, in1, in2, out, dtype, graph, deterministic):
    p = _edge_sum(mul, in1, in2, out, dtype)
    degrees = np.array(DEGREES[graph] if graph != "many" else DEGREES[graph][:90])
    nodes, edges = len(degrees), int(degrees.sum())
    rng = np.random.default_rng(edges)
    rows, cols, _, perm = orc.coord_graph(np.repeat(np.arange(nodes), degrees), rng.integers(0, nodes, edges))
    x, y, dz = (rng.normal(size=(n, r.dim)).astype(dtype) for n, r in ((nodes, p.irreps_in1), (edges, p.irreps_in2), (nodes, p.irreps_out)))
    ones = np.ones((edges, p.weight_numel), dtype)
    want = [orc.conv_forward(p, x, y, ones, rows, cols), *orc.conv_backward(p, x, y, ones, dz, rows, cols)[:2]]
    conv = _UnitWeightConv(p, deterministic)
    index = _cuda(rows, cols) + (_cuda(perm) if deterministic else [])
    plain = None
    for wrap in (lambda t: t, _unaligned):
        xt, yt, dzt = (wrap(t) for t in _cuda(x, y, dz))
        got = [conv.forward(xt, yt, *index), *conv.backward_helper(xt, yt, dzt, *index)]
        conv.internal.check()
        for g, r in zip(got, want):
            assert rel_err(g.cpu().numpy(), r) < REL_TOL[dtype]
        if deterministic and plain is not None:     # copies in pieces or in elements: the same sums
            assert all(torch.equal(a, b) for a, b in zip(got, plain))
        plain = got


def test_large_lists_in_edge_blocks(monkeypatch):
    """Wide rows stay with the slice kernel on lists of every length; with scratch for a part of the edges it runs block by block."""
    monkeypatch.setenv("OEQ_B200_BWD_SCRATCH_MB", "1")
    monkeypatch.setenv("OEQ_B200_BWD_MIN_BLOCK", "1")
    monkeypatch.setenv("OEQ_B200_RECV_MIN_EDGES", "1")
    p = _edge_sum(128, E2, E2, E2)
    nodes, edges, rng = 60, 1500, np.random.default_rng(9)
    rows, cols, _, perm = orc.coord_graph(rng.integers(0, nodes, edges), rng.integers(0, nodes, edges))
    x, y, dz = (rng.normal(size=(n, r.dim)).astype(np.float32) for n, r in ((nodes, p.irreps_in1), (edges, p.irreps_in2), (nodes, p.irreps_out)))
    conv = _UnitWeightConv(p, True)
    dx, dy = conv.backward_helper(*_cuda(x, y, dz, rows, cols, perm))
    conv.internal.check()
    per_block = (1 << 20) // (p.irreps_in1.dim * 4)
    assert conv.internal.last_backward_launches() == 1 + 2 * -(-edges // per_block)
    rx, ry, _ = orc.conv_backward(p, x, y, np.ones((edges, p.weight_numel), np.float32), dz, rows, cols)
    assert rel_err(dx.cpu().numpy(), rx) < REL_TOL[np.float32] and rel_err(dy.cpu().numpy(), ry) < REL_TOL[np.float32]
