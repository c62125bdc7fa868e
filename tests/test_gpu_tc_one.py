"""One-qubit device PTMs on the tensor cores: every place of the target, the
transposed layout, neighbours taken along the outer and the inner axis, partial
tiles, magnitudes that differ from group to group, inf and nan."""
import numpy as np
import pytest
import torch

from conftest import ATOL_F64, RTOL_F64
from quantumsim_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _check(x, p, q, transpose=False):
    got = torch.ops.qsgb.apply_ptm(x, p, [q], L.ARITH_AUTO, 0,
                                   transpose).cpu().numpy()
    m = p.cpu().numpy().T if transpose else p.cpu().numpy()
    xs = np.moveaxis(x.cpu().numpy(), q, 0)
    with np.errstate(invalid='ignore'):  # 0 * inf
        ref = np.moveaxis(np.einsum('rk,k...->r...', m, xs), 0, q)
    # the digits' error is below 2^-49 of the largest product of the row and
    # the group's own four inputs, the reference's four roundings 2^-51
    top = np.abs(m).max(1).reshape((4,) + (1,) * (xs.ndim - 1)) * \
        np.abs(xs).max(0)
    return got, ref, np.moveaxis(top, 0, q) * 2.0 ** -48


@pytest.mark.parametrize('shape,q', [((4,) * 9, q) for q in range(9)] + [
    ((9, 4) + (4,) * 7, 1),       # outer length odd: quarters along z
    ((8, 4) + (4,) * 7, 1),       # outer length 8: two groups of four
    ((4, 4) + (9,) * 5, 1),       # inner length odd
    ((4,) * 3 + (9, 81, 4, 9), 5),
])
@pytest.mark.parametrize('transpose', (False, True))
def test_places(shape, q, transpose):
    rng = np.random.default_rng([q, len(shape), transpose])
    x = torch.from_numpy(rng.standard_normal(shape)).cuda()
    p = torch.from_numpy(rng.standard_normal((4, 4))).cuda()
    got, ref, tol = _check(x, p, q, transpose)
    assert (np.abs(got - ref) <= tol).all()


def test_no_factor_of_four():
    """Neighbours of nine elements only: the general kernel, whose float-float
    rows keep 48 bits (the repository's bound for FP64 rows)."""
    rng = np.random.default_rng(12)
    x = torch.from_numpy(rng.standard_normal((9, 4) + (9,) * 5)).cuda()
    p = torch.from_numpy(rng.standard_normal((4, 4))).cuda()
    got, ref, tol = _check(x, p, 1)
    np.testing.assert_allclose(got, ref, rtol=RTOL_F64,
                               atol=ATOL_F64 * float(tol.max()) * 2.0 ** 48)


@pytest.mark.parametrize('q', (0, 4, 8))
def test_groups_keep_their_own_scale(q):
    """Groups from 2^-900 to 2^900 beside one another, some all zero."""
    rng = np.random.default_rng(q)
    e = rng.integers(-900, 900, size=(4,) * 8)
    xs = rng.standard_normal((4,) * 9) * np.exp2(e.astype(float))
    xs[:, e % 7 == 0] = 0.0
    x = torch.from_numpy(np.ascontiguousarray(np.moveaxis(xs, 0, q))).cuda()
    p = torch.from_numpy(rng.standard_normal((4, 4))).cuda()
    got, ref, tol = _check(x, p, q)
    assert (np.abs(got - ref) <= tol).all()


@pytest.mark.parametrize('value', (np.inf, -np.inf, np.nan))
@pytest.mark.parametrize('q', (0, 4, 8))
def test_inf_and_nan_stay_in_their_group(q, value):
    rng = np.random.default_rng(7)
    xs = rng.standard_normal((4,) * 9)
    xs[2, 1, 3, 0, 2, 1, 0, 3, 1] = value
    x = torch.from_numpy(np.ascontiguousarray(np.moveaxis(xs, 0, q))).cuda()
    p = torch.from_numpy(rng.standard_normal((4, 4))).cuda()
    got, ref, tol = _check(x, p, q)
    bad = ~np.isfinite(ref)
    assert bad.sum() == 4
    assert np.array_equal(got[bad], ref[bad], equal_nan=True)
    assert (np.abs(got[~bad] - ref[~bad]) <= tol[~bad]).all()
