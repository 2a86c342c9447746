"""``TensorProductConv``: fused gather - tensor product - scatter graph convolution.

``Z[n] = sum over edges e with rows[e] == n of TP(X[cols[e]], Y[e], W[e])``.

Mirrors the reference's ``oeq.TensorProductConv`` / ``LoopUnrollConv``
(reference: openequivariance/implementations/convolution/TensorProductConv.py:3-10,
LoopUnrollConv.py:7-87, ConvolutionBase.py:45-109, 560-709):

* ``conv = TensorProductConv(problem, torch_op=True, deterministic=False)``;
  ``Z = conv.forward(X, Y, W, rows, cols)`` for edges in any order (atomic
  accumulation), or, with ``deterministic=True``,
  ``conv.forward(X, Y, W, rows, cols, sender_perm)`` for edges sorted by
  receiver, where ``sender_perm[k]`` is the position in that sorted list of the
  k-th edge in (sender, receiver) order.  The deterministic variant is
  bit-reproducible run to run.
* "uvu" problems whose second input has multiplicity 1 everywhere, per-edge
  weights, int64 indices.
* "uvw" problems with *shared* weights (second input of multiplicity 1), which the reference does not
  offer ("coming soon", reference: README.md:82-85): the dense weight contraction is linear, so the
  per-edge products are summed per receiver first (the fused gather - product - scatter kernel with every
  weight 1) and the weights are applied once per node, on the tensor cores, instead of once per edge
  (``UVWConvPlan``).
* first and second derivatives as ``torch.library`` custom ops.

Unlike the reference, the deterministic backward pass reads the sender and the
receiver of the k-th edge through ``sender_perm[k]``, so it is also correct
for edge lists that are not structurally symmetric.
"""

import itertools

import numpy as np
import torch

from . import _native
from .problem import TPProblem
from .tensor_product import TensorProductBase, _require_cuda, _torch, _torch_dtype

_conv_ids = itertools.count()


class CoordGraph:
    """Canonical edge order of a graph: edges sorted by (row, col), plus the
    permutation that visits them in (col, row) order (reference:
    ConvolutionBase.py:45-70)."""

    def __init__(self, coords, rows, cols, name):
        assert len(rows) == len(cols)
        rows, cols = np.asarray(rows), np.asarray(cols)
        self.nnz = len(rows)
        self.node_count = coords.shape[0]
        self.coords = coords
        self.name = name
        order = np.lexsort((cols, rows))
        self.rows = rows[order]
        self.cols = cols[order]
        self.transpose_perm = np.lexsort((self.rows, self.cols)).astype(self.rows.dtype)


class UVWConvPlan:
    """How a shared-weight "uvw" convolution is split in two fused stages.

    ``Z[n, w, k] = sum_e pw_p sum_u W_p[u, w] sum_ij C_ijk x[s_e, u, i] y[e, j]`` is linear in the per-edge
    product, so the edge sum moves inside: stage 1 is the channel-wise ("uvu") convolution with every
    weight 1 and one output block ``mul_u x ir_out`` per instruction, ``S_p[n, u, k] = sum_e sum_ij C_ijk
    x[s_e, u, i] y[e, j]`` (the fused gather - product - scatter kernels, no weight array); stage 2 is the
    batch "uvw" product ``Z[n] = sum_p pw_p W_p . S_p[n]`` over *nodes*, written as ``S_p x 1x0e -> out``
    so that the tensor-core kernels take it (the l x 0 -> l Wigner tensor is the identity / sqrt(2l+1);
    its value is divided out of the path weight).  The weights keep their layout: instruction p has the
    same ``(u, 1, w)`` block in both problems.
    """

    def __init__(self, config: TPProblem):
        from .irreps import Irreps
        from .wigner import wigner_3j
        assert config.shared_weights, "the fused 'uvw' convolution needs shared weights"
        for mul, _ in config.irreps_in2:
            assert mul == 1, "the fused convolution needs multiplicity 1 for every irrep of the second input"
        blocks, edge_instr, dense_instr, dense_pw = [], [], [], []
        for p, ins in enumerate(config.instructions):
            assert ins.connection_mode == "uvw" and ins.has_weight
            mul_u = config.irreps_in1[ins.i_in1].mul
            ir_out = config.irreps_out[ins.i_out].ir
            blocks.append((mul_u, ir_out))
            edge_instr.append((ins.i_in1, ins.i_in2, p, "uvu", True))
            dense_instr.append((p, 0, ins.i_out, "uvw", True))
            identity = float(np.asarray(wigner_3j(ir_out.l, 0, ir_out.l))[0, 0, 0])
            dense_pw.append(ins.path_weight / identity)
        kw = dict(irrep_dtype=config.irrep_dtype, weight_dtype=config.weight_dtype, internal_weights=False)
        self.edge_sum = TPProblem(config.irreps_in1, config.irreps_in2, Irreps(blocks), edge_instr,
                                  shared_weights=False, **kw)
        self.edge_sum.instructions = [i._replace(path_weight=1.0) for i in self.edge_sum.instructions]
        self.dense = TPProblem(Irreps(blocks), "1x0e", config.irreps_out, dense_instr, shared_weights=True, **kw)
        self.dense.instructions = [i._replace(path_weight=w) for i, w in zip(self.dense.instructions, dense_pw)]
        assert self.dense.weight_numel == config.weight_numel


class TensorProductConv(TensorProductBase):
    def __init__(self, config: TPProblem, torch_op: bool = False, deterministic: bool = False,
                 idx_dtype=np.int64):
        super().__init__(config, torch_op=torch_op)
        assert idx_dtype == np.int64, "indices are int64"
        if len(config.instructions) == 0:
            raise ValueError("Tensor product problem has no valid intructions!")
        for mul, _ in self.L2:
            assert mul == 1, "the fused convolution needs multiplicity 1 for every irrep of the second input"
        self.idx_dtype = idx_dtype
        self.deterministic = deterministic
        self.conv_id = next(_conv_ids)
        self._second_replacement = None
        self.workspace_size = 0
        self.workspace_ptr = 0
        self.unit_weights = False
        if all(inst.connection_mode == "uvw" for inst in config.instructions):
            self._setup_uvw(config)
            return
        for inst in config.instructions:
            assert inst.connection_mode == "uvu", "the fused convolution supports 'uvu', or 'uvw' with shared weights"
        assert not config.shared_weights, "the fused convolution needs per-edge weights"
        self.internal = _native.ConvHandle(config, deterministic)
        # The forward pass needs no scratch (node-aligned segmented reduction).  The deterministic backward pass takes
        # optional scratch (one dX row per edge, capped); large scratch is allocated on first use, per device, and kept
        # with the ops (the reference keeps its workspace on the object: ConvolutionBase.py:93-99).
        self.setup_torch_module()

    @staticmethod
    def name():
        return "LoopUnrollConv"

    # ------------------------------------------------------------------ shared-weight 'uvw' convolution

    def _setup_uvw(self, config):
        from .tensor_product import TensorProduct
        self.plan = UVWConvPlan(config)
        self.edge_sum = _UnitWeightConv(self.plan.edge_sum, self.deterministic)
        self.dense = TensorProduct(self.plan.dense, torch_op=True)
        self.internal = self.edge_sum.internal
        self._ones = {}
        edge_sum, dense, conv = self.edge_sum, self.dense, self

        def ones(ref, rows_n):
            key = (ref.device, ref.dtype, rows_n)
            if key not in conv._ones:
                conv._ones = {key: torch.ones((rows_n, 1), dtype=ref.dtype, device=ref.device)}
            return conv._ones[key]

        def forward(L1_in, L2_in, weights, rows, cols, transpose_perm=None):
            index = (rows, cols) if transpose_perm is None or not conv.deterministic else (rows, cols, transpose_perm)
            s = edge_sum.forward(L1_in, L2_in, *index)
            return dense.forward(s, ones(s, s.shape[0]), weights)

        def backward_helper(L1_in, L2_in, weights, L3_grad, rows, cols, transpose_perm=None):
            index = (rows, cols) if transpose_perm is None or not conv.deterministic else (rows, cols, transpose_perm)
            s = edge_sum.forward(L1_in, L2_in, *index)
            ds, _, dw = dense.backward_helper(s, ones(s, s.shape[0]), weights, L3_grad)
            dx, dy = edge_sum.backward_helper(L1_in, L2_in, ds, *index)
            return [dx, dy, dw]

        self.forward = forward
        self.backward_helper = backward_helper

    def check_device_status(self):
        self.internal.check()
        if hasattr(self, "dense"):
            self.dense.check_device_status()

    # ------------------------------------------------------------------ launches

    def _check(self, x, y, w, rows, cols, perm):
        _require_cuda(x, y, w, rows, cols)
        edges = rows.shape[0]
        if x.dim() != 2 or x.shape[1] != self.L1.dim:
            raise ValueError(f"node features must be [nodes, {self.L1.dim}], got {tuple(x.shape)}")
        if tuple(y.shape) != (edges, self.L2.dim):
            raise ValueError(f"edge features must be [{edges}, {self.L2.dim}], got {tuple(y.shape)}")
        if tuple(w.shape) != (edges, self.config.weight_numel):
            raise ValueError(f"weights must be [{edges}, {self.config.weight_numel}], got {tuple(w.shape)}")
        if cols.shape != rows.shape or rows.dim() != 1:
            raise ValueError("rows and cols must be 1-D and of equal length")
        if rows.dtype != torch.int64 or cols.dtype != torch.int64:
            raise ValueError("rows and cols must be int64")
        dt = _torch_dtype(self.irrep_dtype)
        if x.dtype != dt or y.dtype != dt or w.dtype != dt:
            raise ValueError(f"tensors must be {dt}")
        if perm is not None:
            _require_cuda(perm)
            if perm.shape != rows.shape or perm.dtype != torch.int64:
                raise ValueError("sender_perm must be int64 and as long as rows")

    def _forward_impl(self, x, y, w, rows, cols, perm=None, n_out=None):
        """``n_out``: number of output rows when receivers index a different node set than
        senders (a receiver shard of a partitioned graph); defaults to ``x.shape[0]``."""
        self._check(x, y, w, rows, cols, perm)
        x, y, w = x.contiguous(), y.contiguous(), w.contiguous()
        rows, cols = rows.contiguous(), cols.contiguous()
        n_out = x.shape[0] if n_out is None else int(n_out)
        z = torch.empty((n_out, self.L3.dim), dtype=x.dtype, device=x.device)
        with torch.cuda.device(x.device):
            self.internal.forward(n_out, rows.shape[0], x.data_ptr(), y.data_ptr(), w.data_ptr(),
                                  rows.data_ptr(), cols.data_ptr(), z.data_ptr(), 0, 0,
                                  torch.cuda.current_stream().cuda_stream)
        return z

    def _backward_impl(self, x, y, w, dz, rows, cols, perm=None, scratch=True):
        """``scratch=False`` runs the deterministic pass without scratch memory (the sender-order kernel); otherwise it
        takes what the registered ops keep."""
        self._check(x, y, w, rows, cols, perm)
        if self.deterministic and perm is None:
            raise ValueError("the deterministic convolution needs sender_perm")
        x, y, w, dz = x.contiguous(), y.contiguous(), w.contiguous(), dz.contiguous()
        rows, cols = rows.contiguous(), cols.contiguous()
        perm = perm.contiguous() if (perm is not None and self.deterministic) else None   # (held until the launch)
        perm_ptr = 0 if perm is None else perm.data_ptr()
        dx, dy, dw = torch.empty_like(x), torch.empty_like(y), torch.empty_like(w)
        with torch.cuda.device(x.device):
            if scratch:
                self.workspace_size, self.workspace_ptr = _native.conv_gradients(
                    f"conv_forward{self.conv_id}", x.shape[0], rows.shape[0], x.data_ptr(), y.data_ptr(), w.data_ptr(),
                    dz.data_ptr(), 0, 0, 0, rows.data_ptr(), cols.data_ptr(), perm_ptr, dx.data_ptr(), dy.data_ptr(),
                    dw.data_ptr(), 0)
            else:
                self.internal.backward(x.shape[0], rows.shape[0], x.data_ptr(), y.data_ptr(), w.data_ptr(),
                                       dz.data_ptr(), rows.data_ptr(), cols.data_ptr(), perm_ptr, dx.data_ptr(),
                                       dy.data_ptr(), dw.data_ptr(), 0, 0, torch.cuda.current_stream().cuda_stream)
        return dx, dy, dw

    def _has_fused_double_backward(self):
        return self.internal.has_double_backward()

    @property
    def _double_backward_impl(self):
        """``(x, y, w, dz, ex, ey, ew, rows, cols[, perm]) -> (gx, gy, gw, gdz)`` or ``None``.  Autograd runs the same
        launches natively; a replacement that is assigned here is what autograd calls."""
        return self._second_replacement or self._fused_second

    @_double_backward_impl.setter
    def _double_backward_impl(self, replacement):
        self._second_replacement = replacement
        _native.call_second(f"conv_forward{self.conv_id}", True)

    def _fused_second(self, x, y, w, dz, ex, ey, ew, rows, cols, perm=None):
        """Gradients of ``<ex, dX> + <ey, dY> + <ew, dW>`` with respect to (x, y, w, dz) in two fused launches, or
        ``None`` when the library cannot run them here (no scratch memory for the deterministic variant)."""
        self._check(x, y, w, rows, cols, perm)
        if self.deterministic and perm is None:
            raise ValueError("the deterministic convolution needs sender_perm")
        x, y, w, dz, ex, ey, ew = (t.contiguous() for t in (x, y, w, dz, ex, ey, ew))
        rows, cols = rows.contiguous(), cols.contiguous()
        perm = perm.contiguous() if (perm is not None and self.deterministic) else None   # (held until the launch)
        perm_ptr = 0 if perm is None else perm.data_ptr()
        gx, gy, gw, gdz = torch.empty_like(x), torch.empty_like(y), torch.empty_like(w), torch.empty_like(dz)
        with torch.cuda.device(x.device):
            try:
                self.workspace_size, self.workspace_ptr = _native.conv_gradients(
                    f"conv_forward{self.conv_id}", x.shape[0], rows.shape[0], x.data_ptr(), y.data_ptr(), w.data_ptr(),
                    dz.data_ptr(), ex.data_ptr(), ey.data_ptr(), ew.data_ptr(), rows.data_ptr(), cols.data_ptr(), perm_ptr,
                    gx.data_ptr(), gy.data_ptr(), gw.data_ptr(), gdz.data_ptr())
            except _native.OeqError as err:
                if err.code == _native.OEQ_ERR_UNSUPPORTED:
                    return None
                raise
        return gx, gy, gw, gdz

    def exec_conv_rawptrs(self, L1_in, L2_in, weights, L3_out, rows, cols, nnz, node_count, workspace=0,
                          stream=0):
        """Launch on raw device pointers; argument order of the reference's
        ``JITConvImpl.exec_conv_rawptrs`` (extension/convolution.hpp:27-50)."""
        self.internal.forward(int(node_count), int(nnz), int(L1_in), int(L2_in), int(weights), int(rows),
                              int(cols), int(L3_out), workspace, 0, stream)

    def backward_rawptrs(self, L1_in, L1_grad, L2_in, L2_grad, weights, weights_grad, L3_grad, rows, cols, nnz,
                         node_count, workspace=0, transpose_perm=0, stream=0):
        self.internal.backward(int(node_count), int(nnz), int(L1_in), int(L2_in), int(weights), int(L3_grad),
                               int(rows), int(cols), int(transpose_perm), int(L1_grad), int(L2_grad),
                               int(weights_grad), workspace, 0, stream)

    # ------------------------------------------------------------------ torch ops

    def setup_torch_module(self):
        conv, cfg = self, self.config
        index = "Tensor rows, Tensor cols" + (", Tensor transpose_perm" if self.deterministic else "")
        second = f"conv_second{self.conv_id}"
        torch.library.define(f"openequivariance_b200::{second}",
                             "(Tensor x, Tensor y, Tensor w, Tensor dz, Tensor ex, Tensor ey, Tensor ew, "
                             f"{index}) -> Tensor[]")

        @torch.library.impl(f"openequivariance_b200::{second}", "CUDA")
        def _(*args):
            # empty where the library has no fused second derivatives here: the caller composes them
            fused = conv._double_backward_impl(*args) if conv._has_fused_double_backward() else None
            return [] if fused is None else list(fused)

        self.forward, self.backward_helper = _native.register_ops(
            f"conv_forward{self.conv_id}", f"conv_backward{self.conv_id}", self.internal,
            deterministic=self.deterministic, f64=self.irrep_dtype == np.float64,
            dims=(self.L1.dim, self.L2.dim, self.L3.dim, cfg.weight_numel), second=second)

    # ------------------------------------------------------------------ host-array entry points

    def forward_cpu(self, L1_in, L2_in, weights, L3_out, graph):
        """Host arrays and a ``CoordGraph`` in, ``L3_out`` filled in place
        (reference: LoopUnrollConv / ConvolutionBase.forward_cpu, ConvolutionBase.py:104-134)."""
        assert graph.rows.dtype == self.idx_dtype
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
               for a in (L1_in, L2_in, weights, graph.rows, graph.cols)]
        perm = torch.from_numpy(np.ascontiguousarray(graph.transpose_perm)).cuda() if self.deterministic else None
        L3_out[:] = self._forward_impl(*dev, perm).cpu().numpy()

    def backward_cpu(self, L1_in, L1_grad, L2_in, L2_grad, L3_grad, weights, weights_grad, graph):
        assert graph.rows.dtype == self.idx_dtype
        x, y, w, dz, rows, cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
                                   for a in (L1_in, L2_in, weights, L3_grad, graph.rows, graph.cols)]
        perm = torch.from_numpy(np.ascontiguousarray(graph.transpose_perm)).cuda() if self.deterministic else None
        dx, dy, dw = self._backward_impl(x, y, w, dz, rows, cols, perm)
        L1_grad[:] = dx.cpu().numpy()
        L2_grad[:] = dy.cpu().numpy()
        weights_grad[:] = dw.cpu().numpy()


class _UnitWeightConv:
    """The fused gather - product - scatter kernels with every weight 1 and no weight array (first stage of the
    shared-weight "uvw" convolution): ``S = forward(X, Y, rows, cols[, sender_perm])``, first and second
    derivatives with respect to X and Y as custom ops."""

    def __init__(self, problem: TPProblem, deterministic: bool):
        self.config, self.deterministic = problem, deterministic
        self.L1, self.L2, self.L3 = problem.irreps_in1, problem.irreps_in2, problem.irreps_out
        self.conv_id = next(_conv_ids)
        self.internal = _native.ConvHandle(problem, deterministic, unit_weights=True)
        self.forward, self.backward_helper = _native.register_ops(
            f"conv_edge_sum{self.conv_id}", f"conv_edge_sum_backward{self.conv_id}", self.internal,
            deterministic=deterministic, has_weights=False, f64=problem.irrep_dtype == np.float64,
            dims=(self.L1.dim, self.L2.dim, self.L3.dim, 0))


LoopUnrollConv = TensorProductConv
