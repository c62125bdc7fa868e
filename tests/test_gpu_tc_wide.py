"""Dense PTMs larger than 16 x 16 on the tensor cores: every layout, tiles with
one group, a partial last tile and several tiles, strides with the less
significant target last (tiles through shared memory) and not, odd and even
dimensions, rectangular PTMs, FP64 and FP32.

Bound, derived from the split, with at most 81 terms: the fixed point of a row
or group truncates each factor by at most 2^-53 (FP32: 2^-35) of its maximum,
and the digit pairs beyond the last level add at most 5 * 2^-54 (3 * 2^-36) a
term, so FP64 errs by less than 81 * 9 * 2^-54 < 2^-44 of
max_k |P_rk| max_k |x_k| plus the rounding of the result, FP32 by
81 * 7 * 2^-36 < 2^-26 of it plus 2^-24 of the result.  (The digits are finer
than that: 55 and 39 bits.)"""
import zlib

import numpy as np
import pytest
import torch

import quantumsim_gb300 as qg
from quantumsim_gb300 import _lib as L
from quantumsim_gb300 import bases as B
from oracle import pauli_vector_np as O

pytestmark = pytest.mark.gpu

# vector shape, qudits, output dimensions of the qudits
CASES = [
    ((9, 9), (0, 1), (9, 9)),              # one group
    ((9, 9, 9), (1, 2), (9, 9)),           # staged, one partial tile
    ((9, 9, 9), (2, 0), (9, 9)),           # staged, swapped, Y > 1
    ((9, 9, 9, 9), (0, 2), (9, 9)),        # Z = 9
    ((4, 9, 9, 9), (1, 2), (9, 9)),        # one full tile less 92
    ((9, 9, 9, 9, 4), (3, 1), (9, 9)),     # several tiles, Z = 36
    ((9, 9, 9, 9, 9), (4, 0), (9, 9)),     # staged, x and y, several tiles
    ((4, 9, 4, 9), (0, 1), (4, 9)),        # 36 x 36
    ((9, 4, 9, 4), (2, 3), (9, 4)),        # 36 x 36, staged, even run
    ((9, 9, 4), (0, 1), (9, 4)),           # 36 x 81
    ((9, 4, 9, 4), (3, 0), (9, 9)),        # 81 x 36, swapped, staged
]


def _ref(x, p, qudits):
    return O.apply_ptm(x.astype(np.longdouble), p.astype(np.longdouble),
                       *qudits)


def _group_bound(x, p, qudits):
    """max_k |P_rk| max_k |x_k| for every output."""
    k = len(qudits)
    ax = tuple(range(k, 2 * k))
    pm = np.abs(p).max(axis=ax)                       # per row
    xm = np.abs(x).max(axis=tuple(qudits), keepdims=True)
    order = np.argsort(qudits)
    shape = [1] * x.ndim
    for i in order:
        shape[qudits[i]] = pm.shape[i]
    return xm * pm.transpose(order).reshape(shape)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('shape,qudits,dout', CASES)
@pytest.mark.parametrize('where', ['host', 'device', 'transposed'])
def test_wide_dense_ptm(shape, qudits, dout, dtype, where):
    rng = np.random.default_rng(zlib.crc32(repr((shape, qudits)).encode()))
    din = tuple(shape[q] for q in qudits)
    p = rng.standard_normal(dout + din) * np.exp(
        rng.normal(0, 2, dout + (1,) * len(din)))
    x = rng.standard_normal(shape) * np.exp(rng.normal(0, 1, shape))
    xt = torch.from_numpy(x).cuda().to(dtype)
    x = xt.cpu().numpy().astype(np.float64)
    arith = L.ARITH_AUTO if dtype == torch.float64 else L.ARITH_F32
    pt, tr = torch.from_numpy(p), False
    if where == 'transposed':  # the stored matrix is the forward PTM
        k = len(din)
        pt = pt.permute(list(range(k, 2 * k)) + list(range(k))).contiguous()
        tr = True
    if where != 'host':
        pt = pt.cuda()
    got = torch.ops.qsgb.apply_ptm(xt, pt, list(qudits), arith, 0,
                                   tr).cpu().numpy()
    want = _ref(x, p, qudits)
    eps = (2.0 ** -44, 2.0 ** -52) if dtype == torch.float64 else \
        (2.0 ** -26, 2.0 ** -23)
    bound = eps[0] * _group_bound(x, p, qudits) + eps[1] * np.abs(want)
    assert got.shape == want.shape
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize('scale', [1e300, 1e-300, 1e-310, 0.0])
@pytest.mark.parametrize('qudits', [(0, 1), (2, 1)])
def test_wide_range_and_non_finite(scale, qudits):
    """Results outside the normal range, and inf and nan in a group, come from
    the native FP64 recomputation; other groups are not touched by them."""
    rng = np.random.default_rng(5)
    p = rng.standard_normal((9,) * 4)
    x = rng.standard_normal((9, 9, 9)) * scale
    bad = 4
    idx = [3, 3, 3]
    free = ({0, 1, 2} - set(qudits)).pop()
    idx[free] = bad
    for value in (0.5 * scale, np.inf, np.nan):
        x[tuple(idx)] = value
        got = torch.ops.qsgb.apply_ptm(
            torch.from_numpy(x).cuda(), torch.from_numpy(p).cuda(),
            list(qudits), L.ARITH_AUTO, 0, False).cpu().numpy()
        with np.errstate(all='ignore'):
            want = O.apply_ptm(x, p, *qudits)
        gg, ww = np.moveaxis(got, free, 0), np.moveaxis(want, free, 0)
        others = [i for i in range(9) if i != bad]
        bound = 81 * 2.0 ** -44 * np.abs(p).max() * scale + 1e-322 * 1e5
        assert np.all(np.abs(gg[others] - ww[others]) <= bound)
        if np.isfinite(value):
            assert np.all(np.abs(gg[bad] - ww[bad]) <= bound)
        else:
            assert np.array_equal(np.isnan(gg[bad]), np.isnan(ww[bad]))
            assert np.array_equal(np.isinf(gg[bad]), np.isinf(ww[bad]))


def test_sparse_and_selected_arithmetic_keep_their_kernels():
    """'f64' keeps exact IEEE products (equal to the oracle's bound), and the
    public class gives the dense result for every arithmetic."""
    rng = np.random.default_rng(6)
    p = rng.standard_normal((9,) * 4) / 9
    x = rng.standard_normal((9,) * 3)
    want = _ref(x, p, (0, 2))
    mag = _ref(np.abs(x), np.abs(p), (0, 2))
    for arith in ('auto', 'f64', 'df64'):
        pv = qg.PauliVectorGB300([B.general(3)] * 3, x, arith=arith)
        pv.apply_ptm(p, 0, 2)
        assert np.all(np.abs(pv.to_pv() - want) <= 1e-12 * mag)
