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
