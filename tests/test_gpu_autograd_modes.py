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


@pytest.mark.parametrize('which', ('state', 'ptm', 'gradient'))
def test_negated_views(which):
    x = torch.rand(4, 4, 4, device='cuda', dtype=torch.float64)
    p = _rotation()
    w = torch.rand(4, 4, 4, device='cuda', dtype=torch.float64)
    if which == 'state':
        x = torch._neg_view(x)
    elif which == 'ptm':
        p = torch._neg_view(p)
    else:
        w = torch._neg_view(w)
    x.requires_grad_(True)
    p.requires_grad_(True)
    y = A.apply_ptm_diff(x, p, 1)
    gx, gp = torch.autograd.grad(y, (x, p), w)
    want = _applied(x, p)
    wx, wp = torch.autograd.grad(want, (x, p), w)
    for a, b in ((y, want), (gx, wx), (gp, wp)):
        # sums of at most 16 products of values of at most 1
        assert (a - b).abs().max() <= 1e-14


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
