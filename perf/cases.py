"""Workloads of the tensor product and the graph convolution, as programs that use them run them.

The operators are the two that an equivariant network calls: the batch product ``oeq.TensorProduct`` and the fused
graph convolution ``oeq.TensorProductConv``.  A case names

  op         tp | conv
  pass       forward    inference that needs no gradient
             gradients  forward and backward through autograd: a training step on energies, or one step of
                        molecular dynamics, where the forces are the gradient of the energy
             second     forward, gradients that stay in the graph, and the derivative of those: a training step
                        on forces
  problem    the irreps (``PROBLEMS``)
  dtype      f32 | f64 (interatomic potentials are often run in double precision)
  rows                               of a batch product
  nodes, degree, numbering, variant  of a convolution: size and mean degree of a radius graph, node ids sorted in
                                     space or as they come, bit-reproducible or atomic accumulation

``listed`` has the sizes of this repository's benchmark and tests and ordinary ones between; ``draw`` gives others of
the same ranges.
"""

import functools
import math

import numpy as np
import torch

import openequivariance_b200 as oeq
from openequivariance_b200.graph import periodic_radius_graph, spherical_harmonics
from openequivariance_b200.wigner import cg_nonzeros

PROBLEMS = {
    # one l=2 x l=3 -> l=2 path: the first example of the documentation
    "readme": ("tpp", "1x2e", "1x3e", "1x2e"),
    "interaction_8": ("channelwise", "8x0e+8x1o", "1x0e+1x1o", "8x0e+8x1o"),
    "nequip": ("channelwise", "32x0e+32x1o+32x2e", "0e+1o+2e", "32x0e+32x1o+32x2e"),
    "mace": ("channelwise", "128x0e+128x1o+128x2e", "1x0e+1x1o+1x2e+1x3o", "128x0e+128x1o+128x2e"),
    "mace_large": ("channelwise", "128x0e+128x1o+128x2e+128x3o", "1x0e+1x1o+1x2e+1x3o",
                   "128x0e+128x1o+128x2e+128x3o"),
    # dense weights, shared by all rows
    "fc_64": ("fully_connected", "64x0e+64x1o+64x2e", "0e+1o+2e", "64x0e+64x1o+64x2e"),
    # dense weights, one set for each row
    "diffdock": ("fully_connected_rows", "10x1o + 10x1e + 48x0e + 48x0o", "1x0e + 1x1o",
                 "10x1o + 10x1e + 48x0e + 48x0o"),
}


def listed():
    def tp(name, what, problem, rows, dtype="f32"):
        return {"name": name, "op": "tp", "pass": what, "problem": problem, "dtype": dtype, "rows": rows}

    def conv(name, what, problem, nodes, degree, variant, numbering, dtype="f32"):
        return {"name": name, "op": "conv", "pass": what, "problem": problem, "dtype": dtype, "nodes": nodes,
                "degree": degree, "variant": variant, "numbering": numbering}

    return [
        # the documentation's first call: what a call costs when there is almost nothing to compute
        tp("tp_readme_1000", "forward", "readme", 1000),
        # energy and forces of one small molecule: a molecular-dynamics step is a chain of such calls
        conv("conv_mace_molecule", "gradients", "mace", 27, 10.0, "deterministic", "random"),
        # a box of liquid in double precision, as potentials are run where energies have to be conserved
        conv("conv_mace_f64", "gradients", "mace", 1013, 24.0, "atomic", "random", "f64"),
        # inference on a mid-sized structure, atoms in the order of the input file
        conv("conv_nequip_forward", "forward", "nequip", 3001, 37.0, "deterministic", "random"),
        # the benchmark's narrow convolution
        conv("conv_nequip_20k", "gradients", "nequip", 20000, 40.0, "atomic", "morton"),
        # a training batch of structures, on energies
        conv("conv_mace_5k", "gradients", "mace", 4999, 30.0, "deterministic", "morton"),
        # the same on forces: derivatives of the gradients
        conv("conv_mace_forces_2k", "second", "mace", 2003, 28.0, "deterministic", "morton"),
        # the benchmark's wide convolution, at a fifth of its nodes
        conv("conv_mace_large_40k", "gradients", "mace_large", 40000, 30.0, "deterministic", "morton"),
        # dense shared weights in a convolution
        conv("conv_fc64_10k", "gradients", "fc_64", 10007, 40.0, "deterministic", "morton"),
        # the benchmark's batch products: channel-wise, and dense with shared weights
        tp("tp_mace_50k", "gradients", "mace", 50000),
        tp("tp_fc64_100k", "gradients", "fc_64", 100000),
        # dense weights from a network, one set for each edge of a docking pose
        tp("tp_diffdock_2k", "gradients", "diffdock", 2011),
    ]


#: What is drawn: (op, problem, passes, dtypes, most rows or edges in f32).  Double precision takes half as many.
#: The least is 1 row, or a graph of 8 nodes.
RANGES = [
    ("tp", "readme", ("forward", "gradients"), ("f32", "f64"), 100_000),
    ("tp", "nequip", ("forward", "gradients", "second"), ("f32", "f64"), 300_000),
    ("tp", "mace", ("forward", "gradients", "second"), ("f32", "f64"), 60_000),
    ("tp", "fc_64", ("forward", "gradients"), ("f32", "f32", "f64"), 120_000),
    ("tp", "diffdock", ("forward", "gradients"), ("f32",), 20_000),
    ("conv", "interaction_8", ("gradients", "second"), ("f32", "f64"), 400_000),
    ("conv", "nequip", ("forward", "gradients", "second"), ("f32", "f32", "f64"), 1_000_000),
    ("conv", "mace", ("forward", "gradients", "gradients", "second"), ("f32", "f32", "f64"), 600_000),
    ("conv", "mace_large", ("forward", "gradients"), ("f32",), 1_000_000),
    ("conv", "fc_64", ("forward", "gradients"), ("f32",), 800_000),
]


def draw(rng):
    op, problem, passes, dtypes, most = rng.choice(RANGES)
    case = {"op": op, "pass": rng.choice(passes), "problem": problem, "dtype": rng.choice(dtypes)}
    if case["dtype"] == "f64":
        most //= 2
    if op == "tp":
        case["rows"] = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
        return case
    degree = round(rng.uniform(8.0, 60.0), 1)
    nodes = int(round(math.exp(rng.uniform(math.log(8), math.log(most / degree)))))
    case.update(nodes=nodes, degree=min(degree, round(0.4 * nodes, 1)),     # a cutoff within half the box
                variant=rng.choice(("deterministic", "atomic")), numbering=rng.choice(("morton", "random")))
    return case


# ------------------------------------------------------------------------------------------ what a program keeps

@functools.lru_cache(maxsize=None)
def problem_of(name, dtype):
    kind, in1, in2, out = PROBLEMS[name]
    dt = np.float32 if dtype == "f32" else np.float64
    kw = dict(irrep_dtype=dt, weight_dtype=dt)
    if kind == "channelwise":
        return oeq.ChannelwiseTPP(in1, in2, out, **kw)
    if kind == "fully_connected":
        return oeq.FullyConnectedTPProblem(in1, in2, out, **kw)
    if kind == "fully_connected_rows":
        return oeq.FullyConnectedTPProblem(in1, in2, out, shared_weights=False, **kw)
    return oeq.TPProblem(in1, in2, out, [(0, 0, 0, "uvu", True)], shared_weights=False, internal_weights=False, **kw)


@functools.lru_cache(maxsize=None)
def operator(op, name, dtype, variant=None):
    """A network makes its operators once."""
    problem = problem_of(name, dtype)
    if op == "tp":
        return oeq.TensorProduct(problem, torch_op=True)
    return oeq.TensorProductConv(problem, torch_op=True, deterministic=variant == "deterministic")


def neighbours(nodes, degree, numbering, seed):
    """Receivers, senders, sender-order permutation and unit vectors of the ``nodes * degree / 2`` closest pairs of a
    random periodic structure, in both directions: structures of the same size have equally many edges."""
    graph = periodic_radius_graph(nodes, 1.3 * degree + 8.0, seed=seed, numbering=numbering)
    edges = edge_count(nodes, degree)
    delta = graph.coords[graph.cols] - graph.coords[graph.rows]
    lengths = np.linalg.norm(delta - np.round(delta), axis=1)
    near = lengths <= np.partition(lengths, edges - 1)[edges - 1]
    rows, cols = graph.rows[near], graph.cols[near]
    assert len(rows) == edges
    return rows, cols, np.lexsort((rows, cols)), graph.vectors[near]


def edge_count(nodes, degree):
    return 2 * int(nodes * degree / 2)


def prepare(case, seed):
    problem = problem_of(case["problem"], case["dtype"])
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return torch.randn(*shape, device="cuda", dtype=dt, generator=gen).mul_(scale)

    lmax = max(ir.l for _, ir in problem.irreps_in2)
    index = ()
    if case["op"] == "tp":
        n_in = n_out = edges = case["rows"]
        vectors = torch.nn.functional.normalize(normal(edges, 3), dim=1)
    else:
        rows, cols, sender_perm, vectors = neighbours(case["nodes"], case["degree"], case["numbering"], seed)
        n_in = n_out = case["nodes"]
        edges = len(rows)
        vectors = torch.from_numpy(vectors).cuda().to(dt)
        index = (rows, cols) + ((sender_perm,) if case["variant"] == "deterministic" else ())
        index = tuple(torch.from_numpy(a).cuda() for a in index)
    # edge attributes: spherical harmonics of the edge directions
    y = spherical_harmonics(lmax, vectors)
    if y.shape[1] != problem.irreps_in2.dim:          # a single l
        y = y[:, -problem.irreps_in2.dim:]
    y = y.contiguous()
    w = (normal(problem.weight_numel, scale=0.125) if problem.shared_weights
         else normal(edges, problem.weight_numel))
    state = {"call": operator(case["op"], case["problem"], case["dtype"], case.get("variant")).forward,
             "pass": case["pass"], "inputs": (normal(n_in, problem.irreps_in1.dim), y, w), "index": index}
    if case["pass"] != "forward":
        state["dz"] = normal(n_out, problem.irreps_out.dim)
        for t in state["inputs"]:
            t.requires_grad_(True)
    if case["pass"] == "second":
        state["dz"].requires_grad_(True)              # it comes from the layers behind
        state["cotangents"] = tuple(normal(*t.shape) for t in state["inputs"])
    return state


def run(state):
    inputs, index = state["inputs"], state["index"]
    if state["pass"] == "forward":
        with torch.no_grad():
            return state["call"](*inputs, *index)
    z = state["call"](*inputs, *index)
    if state["pass"] == "gradients":
        return (z.detach(), *torch.autograd.grad(z, inputs, state["dz"]))
    first = torch.autograd.grad(z, inputs, state["dz"], create_graph=True)
    second = torch.autograd.grad(first, (*inputs, state["dz"]), state["cotangents"])
    return (z.detach(), *(g.detach() for g in first), *second)


# ------------------------------------------------------------------------------------------ what a pass must do

@functools.lru_cache(maxsize=None)
def _counts(name):
    """Multiply-adds of one row: (forward, backward, dense weight contraction within the forward)."""
    problem = problem_of(name, "f32")
    fwd = bwd = dense = 0
    for ins in problem.instructions:
        l = [r[i].ir.l for r, i in ((problem.irreps_in1, ins.i_in1), (problem.irreps_in2, ins.i_in2),
                                    (problem.irreps_out, ins.i_out))]
        nz = cg_nonzeros(*l)
        pairs = len({t[:2] for t in nz})
        u, v = ins.path_shape[:2]
        fwd += u * v * (pairs + len(nz))
        bwd += u * v * (3 * pairs + len(nz))
        if ins.connection_mode == "uvw":
            dense += math.prod(ins.path_shape) * (2 * l[2] + 1)
        else:
            fwd += u * v * (2 * l[2] + 1)
    return fwd, bwd, dense


def work(case):
    """Bytes: each call (forward, backward, derivative of the backward) reads its inputs and writes its outputs once.
    Operations: the channel-wise products of every row, and the dense contraction where there is one (in a
    convolution with shared weights once for each node)."""
    problem = problem_of(case["problem"], case["dtype"])
    s = 4 if case["dtype"] == "f32" else 8
    conv = case["op"] == "conv"
    nodes = case["nodes"] if conv else case["rows"]
    edges = edge_count(nodes, case["degree"]) if conv else nodes
    x, z, y = nodes * problem.irreps_in1.dim * s, nodes * problem.irreps_out.dim * s, edges * problem.irreps_in2.dim * s
    w = problem.weight_numel * s * (1 if problem.shared_weights else edges)
    index = edges * 16 if conv else 0
    fwd, bwd, dense = _counts(case["problem"])
    dense *= nodes
    total = x + y + w + z + index
    flops = 2 * (fwd * edges + dense)
    if case["pass"] != "forward":
        total += 2 * (x + y + w) + z + index
        flops += 2 * (bwd * edges + 2 * dense)
    if case["pass"] == "second":
        total += 3 * (x + y + w) + 2 * z + index      # rows and cotangents in, four gradients out
        flops += 4 * (bwd * edges + 2 * dense)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Sums of some hundreds of products in the data type, in another order."""
    return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-13}
