"""The convolution's slice kernels (one warp per 32 channels, two edges of a receiver at a time) at the sizes where
their walk can go wrong: runs of one, two, odd and even numbers of edges around the 32-edge index window, receivers
without edges at both ends and in between, fewer edges than walkers, rows that break the 16-byte rule; one slice of a
full or partly filled warp and several slices."""
import numpy as np
import pytest
import torch

import openequivariance_b200 as oeq
from oracle import tp_oracle as orc
from conftest import problem_by_name
from helpers import REL_TOL, conv_inputs, rel_err

pytestmark = pytest.mark.gpu

DEGREES = {
    "runs": [0, 0, 1, 2, 3, 0, 30, 31, 32, 33, 0, 61, 62, 63, 64, 5, 0],
    "one_edge": [0, 1, 0],
    "one_run": [0, 1000],
    "many": [7, 8, 0, 9, 16, 17] * 60,
}


def _unaligned(t):
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    view = buf[1:].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("deterministic", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("name,dtype", [("interaction_8", np.float32), ("cw_mixed", np.float64), ("nequip_32", np.float32),
                                        ("nequip_32", np.float64), ("mace_128", np.float32), ("mace_large_128", np.float32)])
@pytest.mark.parametrize("graph", sorted(DEGREES))
def test_walk(name, dtype, graph, deterministic):
    _check_walk(problem_by_name(name, irrep_dtype=dtype, weight_dtype=dtype), dtype, graph, deterministic)


# eight warps per SM, twelve (two estimates), sixteen
NARROW = [("16x0e+16x1o+16x2e", "0e+1o+2e", "16x0e+16x1o+16x2e"), ("8x0e+8x1o", "0e+1o+2e", "8x0e+8x1o+8x2e"),
          ("8x0e+8x1o+8x2e", "0e+1o+2e+3o", "8x0e+8x1o"), ("8x0e+8x1o+8x2e", "0e+1o", "8x0e+8x1o+8x2e")]


@pytest.mark.parametrize("deterministic", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("irreps", NARROW, ids=[" ".join(i) for i in NARROW])
def test_narrow_double_rows(irreps, deterministic):
    p = oeq.ChannelwiseTPP(*irreps, irrep_dtype=np.float64, weight_dtype=np.float64)
    _check_walk(p, np.float64, "many", deterministic)


def _check_walk(p, dtype, graph, deterministic):
    degrees = np.array(DEGREES[graph])
    nodes, edges = len(degrees), int(degrees.sum())
    rng = np.random.default_rng(edges)
    rows, cols, _, perm = orc.coord_graph(np.repeat(np.arange(nodes), degrees), rng.integers(0, nodes, edges))
    arrays = conv_inputs(p, nodes, edges, 7)
    x, y, w, dz = (torch.from_numpy(a).cuda() for a in arrays)
    index = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in ((rows, cols, perm) if deterministic else (rows, cols))]
    conv = oeq.TensorProductConv(p, torch_op=True, deterministic=deterministic)
    want = [orc.conv_forward(p, *arrays[:3], rows, cols), *orc.conv_backward(p, *arrays, rows, cols)]
    plain = None
    for wrap in (lambda t: t, _unaligned):
        ins = [wrap(t) for t in (x, y, w, dz)]
        got = [conv.forward(*ins[:3], *index), *conv.backward_helper(*ins, *index)]
        conv.check_device_status()
        for g, r in zip(got, want):
            assert rel_err(g.cpu().numpy(), r) < REL_TOL[dtype]
        if deterministic and plain is not None:     # copies in pieces or in elements: the same sums
            assert all(torch.equal(a, b) for a, b in zip(got, plain))
        plain = got


@pytest.mark.parametrize("deterministic", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("name", ["nequip_32", "mace_128"])
def test_missing_second_edge(name, deterministic):
    """Receivers with an odd number of edges: the place of the edge that is not there holds zeros, not what an earlier edge
    left there (infinities and NaN of other receivers stay where they belong)."""
    p = problem_by_name(name, irrep_dtype=np.float32, weight_dtype=np.float32)
    degrees = np.array([2, 1, 4, 3, 2, 1, 1, 5] * 40)
    nodes, edges = len(degrees), int(degrees.sum())
    rng = np.random.default_rng(3)
    rows, cols, _, perm = orc.coord_graph(np.repeat(np.arange(nodes), degrees), rng.integers(0, nodes, edges))
    x, y, w, _ = conv_inputs(p, nodes, edges, 11)
    want = orc.conv_forward(p, x, y, w, rows, cols)
    w, y = w.copy(), y.copy()
    bad = degrees[rows] == 2
    w[bad] = np.nan
    y[bad] = np.inf
    index = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in ((rows, cols, perm) if deterministic else (rows, cols))]
    conv = oeq.TensorProductConv(p, torch_op=True, deterministic=deterministic)
    got = conv.forward(*(torch.from_numpy(a).cuda() for a in (x, y, w)), *index).cpu().numpy()
    assert rel_err(got[degrees != 2], want[degrees != 2]) < REL_TOL[np.float32]
    assert np.isnan(got[degrees == 2]).all()
