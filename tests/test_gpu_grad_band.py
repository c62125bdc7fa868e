"""One-qudit PTM gradients with some values outside the float-float band: their
groups alone are multiplied in FP64.

Tolerance: as for all these gradients, 2^-40 of the sum of the absolute
products with at most four groups a thread (their low parts, rounded to 24 bits,
add less than 2^-42 of it), and FP64 sums of fewer than 2^10 partial sums at
2^-53 each."""
import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [np.float64, np.float32])
@pytest.mark.parametrize('groups', [1, 31, 33, 257, 100003])
@pytest.mark.parametrize('kin,kout', [(4, 4), (3, 2)])
@pytest.mark.parametrize('share', ['first', 'last', 'few', 'all'])
@pytest.mark.parametrize('value', [6e-33, 3e30])
def test_groups_outside_the_band(groups, kin, kout, share, value, dtype):
    rng = np.random.default_rng([groups, kin])
    x = rng.normal(size=(groups, kin)).astype(dtype)
    g = rng.normal(size=(groups, kout)).astype(dtype)
    at = {'first': [0], 'last': [groups - 1],
          'few': np.flatnonzero(rng.random(groups) < 0.01),
          'all': np.arange(groups)}[share]
    x[at, kin - 1] *= dtype(value)
    g[at[:1], 0] *= dtype(value)
    ref = g.T.astype(np.float64) @ x.astype(np.float64)
    mag = np.abs(g.T.astype(np.float64)) @ np.abs(x.astype(np.float64))
    for q, (a, b) in ((1, (x, g)), (0, (x.T.copy(), g.T.copy()))):
        got = torch.ops.qsgb.ptm_grad(
            torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(),
            [q]).cpu().numpy()
        excess = float(np.max(np.abs(got - ref) - 2.0 ** -40 * mag))
        assert excess <= 0
