"""Kernels launched as programmatic dependents start while their predecessor
ends: a chain of every apply kernel (specialised, tensor cores, dense device
PTM, wide, generic) and PTM gradients, queued without a wait, eagerly and as a
captured graph, gives bit for bit what the same chain gives with a
synchronisation after every launch."""
import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)

pytestmark = pytest.mark.gpu


def _chain(shape, dtype, seed, count):
    """[(ptm tensor, qudits)]: square PTMs, host and device, sparse and dense."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        k = 1 + i % 2
        qs = [int(q) for q in rng.choice(len(shape), k, replace=False)]
        d = tuple(shape[q] for q in qs)
        n = int(np.prod(d))
        p = np.linalg.qr(rng.standard_normal((n, n)))[0]
        if i % 3 == 0:
            p = np.where(rng.random((n, n)) < 0.25, p, 0.0) + 0.5 * np.eye(n)
        t = torch.from_numpy(p.reshape(d + d).copy())
        out.append((t.cuda() if i % 4 == 3 or t.numel() > 1024 else t, qs))
    return out


def _run(x, chain, arith, sync):
    grads = []
    for ptm, qs in chain:
        y = torch.ops.qsgb.apply_ptm(x, ptm, qs, arith, 0, False)
        if sync:
            torch.cuda.synchronize()
        grads.append(torch.ops.qsgb.ptm_grad(x, y, qs))
        if sync:
            torch.cuda.synchronize()
        x = y
    return [x] + grads


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('shape', [(4,) * 3, (4,) * 6, (4,) * 9, (9,) * 3,
                                   (9, 4, 9, 4)])
def test_queued_chain_equals_synchronised_chain(shape, dtype):
    arith = 0 if dtype == torch.float64 else 3
    rng = np.random.default_rng(1)
    x = torch.from_numpy(rng.standard_normal(shape)).cuda().to(dtype)
    chain = _chain(shape, dtype, 2, 40)
    want = _run(x, chain, arith, True)
    for _ in range(3):
        got = _run(x, chain, arith, False)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            out = _run(x, chain, arith, False)
    torch.cuda.current_stream().wait_stream(stream)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))
