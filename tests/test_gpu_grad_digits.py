"""The digits of the 16 x 16 PTM gradient, to their last level: two groups whose
products nearly cancel, zeros in all others, so that the result shows the lowest
bits of the sum.

Bound: the values have 53 bits within 2 bits of their row's largest, so the 55-bit
digits hold them exactly.  The recombined integer has the unit 2^(er + ek - 54), er
and ek the exponents of the row's and the column's largest value; its last two
levels are shifted down by 14 bits, which takes less than one unit, and the digit
pairs beyond the last level add less than 2 * 5 * 2^14 * 2^-22 units: 1.1 in all.
(Without the last level the errors here would reach several units, without the two
last ones hundreds.)"""
from fractions import Fraction

import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)

pytestmark = pytest.mark.gpu


def _limit():
    """Groups up to which the chunks have 16, above it 32."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return sms * 2 * 8 * 16


def _case(n, a, b, rng):
    x, g = np.zeros((2, 16, n))
    x[:, a] = rng.uniform(1.0, 2.0, 16) * np.exp2(rng.integers(-9, 9, 16))
    x[:, b] = x[:, a]
    g[:, a] = rng.uniform(1.5, 2.0, 16) * np.exp2(rng.integers(-9, 9, 16))
    g[:, b] = -g[:, a] * (1 - rng.uniform(2.0 ** -30, 2.0 ** -20, 16))
    return x, g


# both groups in one chunk of 16, in the halves of one of 32, in the last one
@pytest.mark.parametrize('n,a,b', [(16, 0, 15), (40, 33, 39), (1000, 500, 501),
                                   ('above', 0, 31), ('above', 17, 3),
                                   ('above', -1, -2)])
@pytest.mark.parametrize('place', ['first', 'last'])
def test_near_cancellation(n, a, b, place):
    n = _limit() + 21 if n == 'above' else n
    rng = np.random.default_rng([n, place == 'last'])
    worst = 0.0
    for _ in range(3):
        x, g = _case(n, a, b, rng)
        t = [torch.from_numpy(v).cuda() for v in (x, g)]
        if place == 'first':
            got = torch.ops.qsgb.ptm_grad(*(v.view(4, 4, n) for v in t),
                                          [0, 1])
        else:
            got = torch.ops.qsgb.ptm_grad(
                *(v.t().contiguous().view(n, 4, 4) for v in t), [1, 2])
        got = got.cpu().numpy().reshape(16, 16)
        for r in range(16):
            for k in range(16):
                exact = sum(Fraction(float(g[r, i])) * Fraction(float(x[k, i]))
                            for i in (a, b))
                er, ek = (int(np.floor(np.log2(np.abs(v).max())))
                          for v in (g[r], x[k]))
                unit = Fraction(2) ** (er + ek - 54)
                worst = max(worst, float(abs(Fraction(float(got[r, k])) -
                                             exact) / unit))
    assert worst <= 1.1
