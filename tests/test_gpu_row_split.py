"""Small vectors: the specialised kernels give an item's rows to several
threads.  Every position and layout against the oracle, with groups whose
values leave the float pair's range (each thread recomputes its own rows in
native FP64), and the sizes around which the split changes.

Bound per output as in test_gpu_df_arith.py: (K + 4) 2^-46 sum |P||x|."""
import zlib

import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)
from quantumsim_gb300 import _lib as L
from quantumsim_gb300 import workloads as W
from oracle import pauli_vector_np as O

pytestmark = pytest.mark.gpu


def _ptm(kind, dims, rng):
    n = int(np.prod(dims))
    if kind == 'dense':
        p = rng.standard_normal((n, n))
    elif kind == 'sparse':
        p = np.where(rng.random((n, n)) < 3.0 / n, rng.standard_normal((n, n)),
                     0.0)
        p[n // 2] = 0.0  # an empty row
    else:  # physical
        if dims == (4,):
            return W.noisy_1q(rng, 3e-5, 2e-5)
        if dims == (4, 4):
            return W.noisy_cz(rng, (0, 1), [3e-5] * 2, [2e-5] * 2)
        if dims == (9,):
            return W.qutrit_1q(rng)
        if dims == (9, 9):
            return W.qutrit_2q(rng)
        p = np.eye(n)
    return p.reshape(dims + dims)


@pytest.mark.parametrize('shape,qudits', [
    ((4,), (0,)), ((4, 4), (0, 1)), ((4, 4), (1, 0)), ((4,) * 4, (1, 2)),
    ((4,) * 4, (3, 0)), ((4,) * 5, (2,)), ((4,) * 7, (1, 4)),
    ((4,) * 8, (6, 7)), ((4,) * 9, (5, 2)), ((4,) * 9, (8,)),
    ((4,) * 10, (3, 7)), ((9, 9), (0, 1)), ((9, 9, 9), (2, 0)),
    ((9, 9, 9), (1,)), ((9, 4, 9), (0, 1)), ((3, 4, 4), (1, 2)),
    ((4, 4, 2), (0, 1))])
@pytest.mark.parametrize('kind', ['physical', 'sparse', 'dense'])
@pytest.mark.parametrize('arith', [L.ARITH_AUTO, L.ARITH_DF64, L.ARITH_F64])
@pytest.mark.parametrize('transpose', [False, True])
def test_small_vectors_every_row(shape, qudits, kind, arith, transpose):
    dims = tuple(shape[q] for q in qudits)
    rng = np.random.default_rng(
        zlib.crc32(repr((shape, qudits, kind)).encode()))
    p = _ptm(kind, dims, rng)
    x = rng.standard_normal(shape)
    free = [i for i in range(len(shape)) if i not in qudits]
    if free:  # two groups outside the float pair's range
        for scale in (1e200, 1e-200):
            idx = [slice(None)] * len(shape)
            for i in free:
                idx[i] = int(rng.integers(shape[i]))
            x[tuple(idx)] *= scale
    got = torch.ops.qsgb.apply_ptm(
        torch.from_numpy(x).cuda(), torch.from_numpy(p), list(qudits), arith,
        0, transpose).cpu().numpy()
    k = len(dims)
    op = p.transpose(list(range(k, 2 * k)) + list(range(k))) if transpose \
        else p
    # entries up to 2^-52 of the largest are residue that the kernels leave out,
    # native FP64 aside
    kept = op if arith == L.ARITH_F64 else np.where(
        np.abs(op) > 2.0 ** -52 * np.abs(op).max(), op, 0.0)
    want = O.apply_ptm(x, kept, *qudits)
    n = int(np.prod(dims))
    bound = (n + 4) * 2.0 ** -46 * O.apply_ptm(np.abs(x), np.abs(op), *qudits)
    if n > 4 and kind == 'dense':
        # the tensor cores' bound: the largest entries of the row and group
        bound = bound + n * 2.0 ** -46 * np.abs(p).max() * np.abs(x).max(
            axis=tuple(qudits), keepdims=True)
    assert np.all(np.abs(got - want) <= bound + 1e-300)
