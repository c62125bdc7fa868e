"""Calls made in ways of their own."""
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import ROOT
import quantumsim_gb300 as qg
from quantumsim_gb300 import bases as B

pytestmark = pytest.mark.gpu


def _ptm(k, seed):
    return torch.from_numpy(np.random.default_rng(seed).normal(
        size=(4,) * (2 * k)))


@pytest.mark.parametrize('qs', [(1,), (0, 2), (2, 0)])
@pytest.mark.parametrize('where', ['cpu', 'cuda'])
def test_batched_gradients(qs, where):
    """is_grads_batched: the backward pass runs on a batch of gradients."""
    x = torch.randn(4, 4, 4, dtype=torch.float64, device='cuda',
                    requires_grad=True)
    p = _ptm(len(qs), 1).to(where).requires_grad_(True)
    y = qg.apply_ptm_diff(x, p, *qs)
    gs = torch.randn(3, *y.shape, dtype=torch.float64, device='cuda')
    got = torch.autograd.grad(y, (x, p), gs, is_grads_batched=True,
                              retain_graph=True)
    for i in range(3):
        want = torch.autograd.grad(y, (x, p), gs[i], retain_graph=True)
        for a, b in zip(got, want):
            assert torch.equal(a[i], b)


def test_under_a_default_device():
    """Page-locked buffers are made on the host whatever the default device."""
    import threading
    fails = []

    def work():  # a new thread: its buffers are made here
        try:
            with torch.device('cuda'):
                pv = qg.PauliVectorGB300([B.general(2)] * 3)
                assert pv.diagonal()[0] == 1.0 and pv.trace() == 1.0
                assert pv.exp_value('ZIZ') == 1.0
                pv.apply_ptm(np.random.default_rng(0).normal(
                    size=(4,) * 4), 0, 1)
                x = pv.data.clone().requires_grad_(True)
                p = _ptm(2, 2).cpu().requires_grad_(True)
                y = qg.apply_ptm_diff(x, p, 0, 2)
                gx, gp = torch.autograd.grad((y * y).sum(), (x, p))
                assert not gp.is_cuda and gx.is_cuda
        except Exception as e:  # handed to the test's thread
            fails.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    if fails:
        raise fails[0]


def test_negated_vector():
    """A vector given as a lazily negated view has the values of the view."""
    t = torch.randn(4, 4, 4, dtype=torch.float64, device='cuda')
    bases = [B.general(2)] * 3
    a, b = (qg.PauliVectorGB300(bases, v) for v in (torch._neg_view(t), -t))
    for _ in range(2):
        np.testing.assert_array_equal(a.diagonal(), b.diagonal())
        np.testing.assert_array_equal(a.to_pv(), b.to_pv())
        assert a.exp_value('XZI') == b.exp_value('XZI')
        assert a.trace() == b.trace()
        for v in (a, b):
            v.apply_ptm(_ptm(2, 3).numpy(), 0, 2)


REFUSED = """
import torch
import quantumsim_gb300

x = torch.randn(4, 4, 4, dtype=torch.float64, device='cuda')
p = torch.randn(4, 4, dtype=torch.float64).cuda()
torch.ops.qsgb.apply_ptm(x, p, [1], 0, 16, False)
torch.cuda.synchronize()


def refused(f):
    try:
        f()
    except RuntimeError:
        return
    raise SystemExit('not refused')


graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
with torch.cuda.stream(stream):
    graph.capture_begin()
    refused(stream.synchronize)  # not allowed: invalidates the capture
    refused(lambda: torch.ops.qsgb.apply_ptm(x, p, [1], 0, 16, False))
    refused(graph.capture_end)
torch.cuda.synchronize()
got = torch.ops.qsgb.take_axis(x, 1, [2, 0])
assert torch.equal(got, x[:, [2, 0]])
print('fine')
"""


def test_refused_launch_leaves_no_error_behind():
    """A launch into a capture that has been invalidated is refused; the next
    launch, which is fine, does not report its error.  (A process of its own:
    torch's generator does not come back from such a capture.)"""
    r = subprocess.run([sys.executable, '-c', REFUSED], cwd=ROOT, text=True,
                       capture_output=True, timeout=300)
    assert r.returncode == 0 and 'fine' in r.stdout, r.stderr[-2000:]
