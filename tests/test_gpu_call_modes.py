"""Calls made in ways of their own."""
import numpy as np
import pytest
import torch

import quantumsim_gb300 as qg
from quantumsim_gb300 import bases as B

pytestmark = pytest.mark.gpu


def _ptm(k, seed):
    return torch.from_numpy(np.random.default_rng(seed).normal(
        size=(4,) * (2 * k)))


def test_refused_launch_leaves_no_error_behind():
    """A launch into a capture that has been invalidated is refused; the next
    launch, which is fine, does not report its error."""
    x = torch.randn(4, 4, 4, dtype=torch.float64, device='cuda')
    p = _ptm(1, 4).cuda()
    torch.ops.qsgb.apply_ptm(x, p, [1], 0, 16, False)
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        try:
            with pytest.raises(RuntimeError):
                stream.synchronize()  # not allowed: invalidates the capture
            with pytest.raises(RuntimeError):
                torch.ops.qsgb.apply_ptm(x, p, [1], 0, 16, False)
            with pytest.raises(RuntimeError):
                graph.capture_end()
        finally:
            del graph
    torch.cuda.synchronize()
    got = torch.ops.qsgb.take_axis(x, 1, [2, 0])
    assert torch.equal(got, x[:, [2, 0]])
