"""Components far below the largest of their group keep their own precision
where no digit split is used (one-qubit device PTMs, gradients of FP32 vectors)
and where a PTM larger than 16 x 16 has zeros.

Bounds are per component, against sums of magnitudes: native FP64 rows of four
terms err by less than 2^-45 of sum |P| |x|, float-float ones by less than the
repository's bound for FP64 rows; FP32 rows of K terms by (K + 2) 2^-24 of it
(entry and product roundings, K sums); a float-float gradient of up to 2^11 groups by
2^-40 of sum |g| |x|, plus 2^-149 a product below the float range."""
import numpy as np
import pytest
import torch

from conftest import RTOL_F64
from quantumsim_gb300 import _lib as L
from oracle import pauli_vector_np as O

pytestmark = pytest.mark.gpu


def _bounded(got, x, p, qs, eps):
    """|got - P x| <= eps |P| |x|, every component (the reference's own
    roundings, 2^-53 a term, are a small part of eps)."""
    ref = O.apply_ptm(x, p, *qs)
    mag = O.apply_ptm(np.abs(x), np.abs(p), *qs)
    excess = float(np.max(np.abs(got - ref) - eps * mag))
    assert excess <= 0


@pytest.mark.parametrize('size', [1e-8, 1e-12, 1e-17, 1e-40])
@pytest.mark.parametrize('n,q', [(8, 3), (9, 0), (9, 8), (10, 4), (11, 2),
                                 (11, 10)])
def test_one_qubit_device_ptm(n, q, size):
    """A rotation about z with dephasing: coherences beside populations; and
    a row whose large entry meets a zero."""
    eps = 2.0 ** -45 if n <= 10 else RTOL_F64
    rng = np.random.default_rng([n, q])
    x = rng.uniform(0.2, 0.8, (4,) * n)
    at = [slice(None)] * n
    for k in (2, 3):
        at[q] = k
        x[tuple(at)] *= size
    c, s = np.cos(0.7) * 0.99, np.sin(0.7) * 0.99
    rot = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, c, -s], [0, 0, s, c]])
    xt = torch.from_numpy(x).cuda()
    for p in (rot, rot.T):
        got = torch.ops.qsgb.apply_ptm(xt, torch.from_numpy(p.copy()).cuda(),
                                       [q], L.ARITH_AUTO, 0, False)
        _bounded(got.cpu().numpy(), x, p, (q,), eps)
    at[q] = 0
    x[tuple(at)] = 0.0
    p = np.full((4, 4), 1e-10) * rng.uniform(0.5, 1, (4, 4))
    p[:, 0] = 1.0
    got = torch.ops.qsgb.apply_ptm(torch.from_numpy(x).cuda(),
                                   torch.from_numpy(p).cuda(), [q],
                                   L.ARITH_AUTO, 0, False)
    _bounded(got.cpu().numpy(), x, p, (q,), eps)


@pytest.mark.parametrize('n', [1, 17, 300, 2048])
@pytest.mark.parametrize('place', ['first', 'last', 'around'])
@pytest.mark.parametrize('gap', [2.0 ** -40, 2.0 ** -60])
def test_gradient_of_fp32_vectors(n, place, gap):
    """Groups where the state is large and the gradient small, and the other
    way round."""
    torch.manual_seed(n)
    x, g = (torch.rand(16, n, dtype=torch.float64) + 0.5 for _ in range(2))
    x[:, 0::2] *= gap
    g[:, 1::2] *= gap
    x, g = x.float(), g.float()
    xs, gs = x.double().numpy(), g.double().numpy()
    ref, mag = gs @ xs.T, np.abs(gs) @ np.abs(xs).T
    shape, qs, perm = {
        'first': ((4, 4, n), (0, 1), (0, 1, 2)),
        'last': ((4, 4, n), (1, 2), (2, 0, 1)),
        'around': ((4, 4, n), (0, 2), (0, 2, 1))}[place]
    x, g = (t.reshape(shape).permute(perm).contiguous().cuda()
            for t in (x, g))
    got = torch.ops.qsgb.ptm_grad(x, g, list(qs)).cpu().numpy().reshape(16, 16)
    excess = float(np.max(np.abs(got - ref) - 2.0 ** -40 * mag))
    assert excess <= n * 2.0 ** -149


SHAPES = [((9, 9), (0, 1)), ((9, 9, 9), (1, 2)), ((9, 9, 9, 4), (2, 0)),
          ((9, 4, 9, 9, 4), (0, 3)), ((4, 9, 9), (0, 2))]


def _with_one_large(shape, qs, small, rng):
    """Values of size `small`; the first component of every group is 1."""
    x = rng.uniform(0.5, 1.0, shape) * small
    at = [slice(None)] * len(shape)
    for q in qs:
        at[q] = 0
    x[tuple(at)] = 1.0
    return x


@pytest.mark.parametrize('shape,qs', SHAPES, ids=str)
@pytest.mark.parametrize('small', [2.0 ** -18, 2.0 ** -30, 2.0 ** -60])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('where', ['host', 'device'])
@pytest.mark.parametrize('hole', ['zero', 'small', None])
def test_wide_ptm(shape, qs, small, dtype, where, hole):
    """The large component enters one row alone, and the others see the small
    ones; or it enters every row, which then has a share of it."""
    rng = np.random.default_rng(len(shape))
    x = _with_one_large(shape, qs, small, rng)
    d = tuple(shape[q] for q in qs)
    k = int(np.prod(d))
    m = rng.uniform(0.5, 1.0, (k, k))
    if hole is not None:  # FP32 rows leave out entries below 2^-30
        m[1:, 0] = 0.0 if hole == 'zero' else \
            2.0 ** -40 if dtype == torch.float64 else 2.0 ** -28
    p = m.reshape(d + d)
    xt = torch.from_numpy(x).cuda().to(dtype)
    x = xt.cpu().numpy().astype(np.float64)
    pt = torch.from_numpy(p)
    arith = L.ARITH_AUTO if dtype == torch.float64 else L.ARITH_F32
    got = torch.ops.qsgb.apply_ptm(xt, pt if where == 'host' else pt.cuda(),
                                   list(qs), arith, 0, False)
    if dtype == torch.float32:
        eps = (k + 2) * 2.0 ** -24
    elif hole is None:  # 81 terms of 9 * 2^-54 of the largest product, half of
        eps = 2.0 ** -42  # which at least is in every sum
    else:
        eps = RTOL_F64
    _bounded(got.cpu().numpy().astype(np.float64), x, p, qs, eps)
