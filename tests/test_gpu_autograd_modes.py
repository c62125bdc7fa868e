"""Autograd functions under create_graph, tracing and negated views."""
import pytest
import torch

import quantumsim_gb300 as qg
from quantumsim_gb300 import autograd as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', (torch.float64, torch.float32))
def test_diagonal_second_derivative(dtype):
    # loss = sum d^3: the gradient of <grad, v> is 6 d v on the diagonal
    b = qg.bases.general(2)
    x = torch.rand(4, 4, 4, device='cuda', dtype=dtype, requires_grad=True)
    v = torch.rand(4, 4, 4, device='cuda', dtype=dtype)
    d = A.diagonal_diff(x, [b] * 3)
    (g,) = torch.autograd.grad((d ** 3).sum(), x, create_graph=True)
    (h,) = torch.autograd.grad((g * v).sum(), x)
    flat = torch.from_numpy(A.diagonal_indices([b] * 3)).cuda()
    want = torch.zeros(64, device='cuda', dtype=torch.float64)
    want[flat] = (6 * x.detach().double() * v.double()).reshape(-1)[flat]
    eps = torch.finfo(dtype).eps  # a few roundings of values below 6
    assert (h.double().reshape(-1) - want).abs().max() <= 32 * eps


def _rotation():
    return torch.tensor([[1., 0, 0, 0], [0, .6, -.8, 0], [0, .8, .6, 0],
                         [0, 0, 0, 1]], dtype=torch.float64)


def _applied(x, ptm):
    return torch.einsum('ab,ibj->iaj', ptm.to(x), x)


@pytest.mark.parametrize('which', (0, 1, 2))
def test_negated_views(which):
    """A lazily negated state, PTM or gradient: the bits of its values."""
    args = [torch.rand(4, 4, 4, device='cuda', dtype=torch.float64),
            _rotation(),
            torch.rand(4, 4, 4, device='cuda', dtype=torch.float64)]
    out = []
    for view in (True, False):
        x, p, w = [t if i != which else torch._neg_view(t) if view else -t
                   for i, t in enumerate(args)]
        x, p = (t.detach().requires_grad_(True) for t in (x, p))
        y = A.apply_ptm_diff(x, p, 1)
        out.append((y,) + torch.autograd.grad(y, (x, p), w))
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_traced_application():
    x, x2 = torch.rand(2, 4, 4, 4, device='cuda', dtype=torch.float64)
    p = _rotation()
    f = torch.jit.trace(lambda t: A.apply_ptm_diff(t, p, 1), (x,),
                        check_trace=False)
    assert (f(x2) - _applied(x2, p)).abs().max() <= 1e-14


def test_traced_by_fx():
    from torch.fx.experimental.proxy_tensor import make_fx
    x, x2 = torch.rand(2, 4, 4, 4, device='cuda', dtype=torch.float64)
    p = _rotation()
    f = make_fx(lambda t: A.apply_ptm_diff(t, p, 1))(x)
    assert (f(x2) - _applied(x2, p)).abs().max() <= 1e-14
