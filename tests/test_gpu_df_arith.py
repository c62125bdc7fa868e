"""Float-float rows of the apply kernels at the edges of their arithmetic:
mantissas where the split rounds up or carries, powers of two, the ends of
the float pair's exponent range, signs that cancel.

Bound per output, derived from the arithmetic: the split of an input and of a
PTM entry err by at most 2^-48 of the value each, the dropped product of the
low words by 2^-48, and each of the row's K accumulation steps rounds terms
of at most 2^-23 of the row's sum of |P||x| four times to 24 bits: together
below (K + 4) 2^-46 sum |P||x|."""
import zlib

import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)
from quantumsim_gb300 import _lib as L
from oracle import pauli_vector_np as O

pytestmark = pytest.mark.gpu


def _from_bits(mant, exp, rng):
    sign = rng.integers(0, 2, mant.size).astype(np.uint64) << np.uint64(63)
    bits = sign | ((exp + 1023).astype(np.uint64) << np.uint64(52)) | mant
    return bits.view(np.float64)


def _mantissas(kind, rng, n):
    m = rng.integers(0, 1 << 52, n).astype(np.uint64)
    if kind == 'ones':          # hi rounds up into the next binade
        return np.full(n, (1 << 52) - 1, dtype=np.uint64)
    if kind == 'powers':
        return np.zeros(n, dtype=np.uint64)
    if kind == 'ties':          # exactly half of hi's last place
        return (m & ~np.uint64((1 << 29) - 1)) | np.uint64(1 << 28)
    if kind == 'below_ties':    # the low word rounds up to that half
        return (m & ~np.uint64((1 << 29) - 1)) | np.uint64((1 << 28) - 1)
    if kind == 'low_ones':      # lo's own rounding carries out of its bits
        return m | np.uint64((1 << 29) - 1)
    return m


@pytest.mark.parametrize('qudits', [(1,), (4,), (0, 3), (4, 2)])
@pytest.mark.parametrize('kind', ['random', 'ones', 'powers', 'ties',
                                  'below_ties', 'low_ones'])
@pytest.mark.parametrize('exps', [(-3, 3), (-102, -95), (120, 127), (0, 0)])
def test_float_float_rows_within_their_bound(qudits, kind, exps):
    rng = np.random.default_rng(zlib.crc32(repr((qudits, kind, exps)).encode()))
    n = 4 ** 5
    x = _from_bits(_mantissas(kind, rng, n),
                   rng.integers(exps[0], exps[1] + 1, n), rng)
    x[rng.integers(0, n, 40)] = 0.0
    x = x.reshape((4,) * 5)
    k = 4 ** len(qudits)
    p = rng.standard_normal((k, k))
    p[:, 1::3] = -p[:, 0:-1:3] if k > 4 else p[:, 1::3]  # cancelling columns
    p = p.reshape((4,) * (2 * len(qudits)))
    got = torch.ops.qsgb.apply_ptm(
        torch.from_numpy(x).cuda(), torch.from_numpy(p), list(qudits),
        L.ARITH_DF64, 0, False).cpu().numpy()
    want = O.apply_ptm(x.astype(np.longdouble), p.astype(np.longdouble),
                       *qudits)
    bound = (k + 4) * 2.0 ** -46 * O.apply_ptm(
        np.abs(x).astype(np.longdouble), np.abs(p).astype(np.longdouble),
        *qudits)
    assert np.all(np.isfinite(got))
    assert np.all(np.abs(got - want) <= bound)
