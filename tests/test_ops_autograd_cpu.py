"""Autograd of the registered ops without a GPU: the nodes (csrc/oeq_torch.cpp) dispatch tensors that are not plain CUDA
tensors through the registered ops, which have CPU kernels here (x * sum(y) * w, trilinear like the product)."""
import pytest
import torch

import openequivariance_b200 as oeq

N = 5


def _forward(x, y, w):
    return x * y.sum(1, keepdim=True) * w


def _gradient(x, y, w, dz):
    s = y.sum(1, keepdim=True)
    return [dz * w * s, (dz * x * w).sum(1, keepdim=True).expand_as(y).contiguous(), dz * x * s]


@pytest.fixture(scope="module")
def product():
    """An operator with x, weight and output rows of 3 values and second-input rows of 3."""
    p = oeq.TPProblem("3x0e", "3x0e", "3x0e", [(0, 0, 0, "uvu", True)], shared_weights=False, internal_weights=False)
    tp = oeq.TensorProduct(p, torch_op=True)
    lib = torch.library.Library("openequivariance_b200", "IMPL")
    lib.impl(f"tp_forward{tp.tp_id}", lambda x, y, w: _forward(x, y, w[:, :3]), "CPU")
    lib.impl(f"tp_grad_helper{tp.tp_id}", lambda x, y, w, dz: [g if g.shape == t.shape else torch.cat([g, torch.zeros(N, 6, dtype=g.dtype)], 1)
                                                             for g, t in zip(_gradient(x, y, w[:, :3], dz), (x, y, w))], "CPU")
    yield tp
    lib._destroy()


def _inputs(grad=True):
    gen = torch.Generator().manual_seed(1)
    x, y, w = (torch.randn(N, k, generator=gen).requires_grad_(grad) for k in (3, 3, 9))
    return x, y, w, torch.randn(N, 3, generator=gen).requires_grad_(grad)


def _wanted(x, y, w, dz):
    return torch.autograd.grad(_forward(x, y, w[:, :3]), (x, y, w), dz)


def test_a_second_pass_without_retained_graph(product):
    """Saved operands are kept with the graph, as the reference's nodes keep them: two backward passes through one result
    need no retain_graph."""
    x, y, w, dz = _inputs()
    z = product.forward(x, y, w)
    for _ in range(2):
        for got, want in zip(torch.autograd.grad(z, (x, y, w), dz.detach()), _wanted(x, y, w, dz.detach())):
            torch.testing.assert_close(got, want)
    first = torch.autograd.grad(z, (x, y, w), dz, create_graph=True)
    for _ in range(2):
        got, = torch.autograd.grad(first[0], y, torch.ones(N, 3))
        want, = torch.autograd.grad(_wanted_graph(x, y, w, dz), y, torch.ones(N, 3))
        torch.testing.assert_close(got, want)


def _wanted_graph(x, y, w, dz):
    return torch.autograd.grad(_forward(x, y, w[:, :3]), x, dz, create_graph=True)[0]


class _NoGradient(torch.autograd.Function):
    """A later layer that returns no gradient for its first input."""

    @staticmethod
    def forward(ctx, z, other):
        return other * 1

    @staticmethod
    def backward(ctx, g):
        return None, g


def test_undefined_gradients_count_as_zeros(product):
    other = torch.ones(2, requires_grad=True)
    x, y, w, dz = _inputs()
    z = product.forward(x, y, w)
    for g, t in zip(torch.autograd.grad(_NoGradient.apply(z, other).sum(), (x, y, w)), (x, y, w)):
        assert g.shape == t.shape and torch.count_nonzero(g) == 0
    first = torch.autograd.grad(z, (x, y, w), dz, create_graph=True)
    for g, t in zip(torch.autograd.grad(_NoGradient.apply(first[1], other).sum(), (x, y, w, dz)), (x, y, w, dz)):
        assert g.shape == t.shape and torch.count_nonzero(g) == 0


@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_is_refused(product, grad):
    """A tangent is not dropped in silence."""
    import torch.autograd.forward_ad as fwad
    x, y, w, dz = _inputs(grad)
    with fwad.dual_level():
        for i in range(3):
            args = [x, y, w]
            args[i] = fwad.make_dual(args[i], torch.ones_like(args[i]))
            with pytest.raises(NotImplementedError, match="forward-mode"):
                product.forward(*args)
            with pytest.raises(NotImplementedError, match="forward-mode"):
                product.backward_helper(*args, dz)
        with pytest.raises(NotImplementedError, match="forward-mode"):
            product.backward_helper(x, y, w, fwad.make_dual(dz, dz.detach()))
    with pytest.raises(NotImplementedError, match="forward-mode"):
        torch.func.jvp(lambda t: product.forward(t, y.detach(), w.detach()), (x.detach(),), (x.detach(),))
    assert torch.isfinite(product.forward(x, y, w)).all()


def test_ops_are_marked_for_compilation(product):
    """torch.compile with only_allow_pt2_compliant_ops takes them."""
    for op in (product.forward, product.backward_helper):
        assert torch.Tag.pt2_compliant_tag in op.tags
