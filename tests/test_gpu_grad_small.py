"""PTM gradients of one qudit with at most four Pauli elements.

A thread multiplies whole groups in float-float, a block with a value outside
the float-float band repeats its groups in FP64.  Reference: numpy float64
sums (pairwise, error far below the bound).

Tolerance: a product is off by at most 2^-46 of itself; a thread adds m groups
and 5 more sums of its warp, whose low parts are rounded to 24 bits of at most
(m + 5) 2^-24 of the absolute sum, m + 5 times: (m + 5)^2 2^-47 of the sum of
the absolute products.  Here m <= 4 (grid of at least 256 blocks at the largest
size; one group per thread below): 2^-40.  Products of values in the band
but below the float range add 2^-149 each.
"""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

import quantumsim_gb300  # noqa: E402,F401

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -40


def reference(x, g, q):
    xk = np.moveaxis(x, q, 0).reshape(x.shape[q], -1).astype(np.float64)
    gr = np.moveaxis(g, q, 0).reshape(g.shape[q], -1).astype(np.float64)
    with np.errstate(invalid='ignore', over='ignore'):
        prod = gr[:, None, :] * xk[None, :, :]
        return prod.sum(-1), np.abs(prod).sum(-1)


def run(x, g, q):
    t = torch.ops.qsgb.ptm_grad(torch.from_numpy(x).cuda(),
                                torch.from_numpy(g).cuda(), [q])
    return t.cpu().numpy()


# bystanders around one warp, one block and many blocks; first, inner and last
# axis; rectangular PTMs
@pytest.mark.parametrize('dtype', [np.float64, np.float32])
@pytest.mark.parametrize('shape,q,kout', [
    ((4,), 0, 4), ((3, 4), 1, 4), ((4, 31), 0, 4), ((4, 33), 0, 3),
    ((5, 4, 51), 1, 1), ((16, 4, 16), 1, 4), ((257, 4), 1, 4),
    ((9, 3, 29), 1, 4), ((7, 2, 9, 4), 1, 2), ((7, 1, 300), 1, 4),
    ((4,) * 10, 4, 4), ((4,) * 10, 9, 4), ((4,) * 9 + (3,), 0, 4)], ids=str)
def test_small_ptm_gradient(shape, q, kout, dtype):
    rng = np.random.default_rng(len(shape) + q)
    x = rng.normal(size=shape).astype(dtype)
    gs = shape[:q] + (kout,) + shape[q + 1:]
    g = (rng.normal(size=gs) * np.exp2(rng.integers(-30, 30, gs))).astype(
        dtype)
    ref, mag = reference(x, g, q)
    got = run(x, g, q)
    assert got.shape == ref.shape
    assert np.all(np.abs(got - ref) <= TOL * mag)


@pytest.mark.parametrize('value', [1e-200, 1e-35, 1e200, np.inf, np.nan])
def test_values_outside_the_band(value):
    rng = np.random.default_rng(1)
    x, g = rng.normal(size=(2, 4, 4, 4, 4, 4, 4, 4))
    x[1, 2, 3, 0, 1, 2, 3] = value
    x[..., 1] = 0.0
    for q in (0, 3, 6):
        ref, mag = reference(x, g, q)
        got = run(x, g, q)
        fin = np.isfinite(ref)
        np.testing.assert_array_equal(np.isfinite(got), fin)
        assert np.all(np.abs(got[fin] - ref[fin]) <= TOL * mag[fin])


@pytest.mark.parametrize('qs,pshape', [((1,), (4, 4)), ((0, 2), (4, 4, 4, 4)),
                                       ((3, 1), (4, 3, 4, 4)),
                                       ((2,), (3, 4))])
def test_host_ptm_gradient_is_the_device_one(qs, pshape):
    """A PTM on the host gets its gradient through page-locked memory while
    the state's is computed: the bits of the same PTM on the device, also
    when it is used twice, and with a graph of the gradient (another path)."""
    rng = np.random.default_rng(len(pshape))
    x = torch.from_numpy(rng.normal(size=(4,) * 5)).cuda()
    p = rng.normal(size=pshape)
    twice = pshape[:len(qs)] == pshape[len(qs):]

    def grads(ptm, **kw):
        a = x.clone().requires_grad_(True)
        y = quantumsim_gb300.apply_ptm_diff(a, ptm, *qs)
        if twice:
            y = quantumsim_gb300.apply_ptm_diff(y, ptm, *qs)
        return torch.autograd.grad((y * y).sum(), [a, ptm], **kw)

    host = torch.from_numpy(p).requires_grad_(True)
    ga, gp = grads(host)
    assert not gp.is_cuda and not gp.is_pinned() and gp.shape == host.shape
    for got, want in zip(grads(host), (ga, gp)):
        assert torch.equal(got, want)
    for got, want in zip(grads(host, create_graph=True), (ga, gp)):
        assert torch.equal(got.detach(), want)
    dev = torch.ops.qsgb.ptm_grad  # one application, the operator's result
    a = x.clone().requires_grad_(True)
    y = quantumsim_gb300.apply_ptm_diff(a, host, *qs)
    g = torch.randn_like(y)
    (gp,) = torch.autograd.grad(y, [host], g)
    assert torch.equal(gp, dev(x, g, list(qs)).cpu())


@pytest.mark.parametrize('n_layers,every', [(1, 1), (3, 8), (4, 2), (5, 2)])
def test_last_segment_kept(n_layers, every):
    """The last segment's states kept or recomputed: the same bits."""
    rng = np.random.default_rng(n_layers)
    ptms = [torch.from_numpy(rng.normal(size=(4, 4, 4, 4))).cuda()
            .requires_grad_(True) for _ in range(n_layers)]
    x = torch.from_numpy(rng.normal(size=(4,) * 4)).cuda().requires_grad_(True)
    calls = []

    def layer(s, i):
        calls.append(i)
        return quantumsim_gb300.apply_ptm_diff(s, ptms[i], i % 3, 3)

    fns = [lambda s, i=i: layer(s, i) for i in range(n_layers)]
    out = []
    for keep in (False, True):
        calls.clear()
        y = quantumsim_gb300.checkpointed(fns, x, every, keep_last=keep)
        out.append([y] + list(torch.autograd.grad((y * y).sum(), [x] + ptms)))
        last = n_layers - (n_layers - 1) // every * every
        assert len(calls) == 2 * n_layers - (last if keep else 0)
    for a, b in zip(*out):
        assert torch.equal(a, b)
