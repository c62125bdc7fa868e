"""Device PTMs of full qubits on FP32 and small FP64 vectors: every width of access (vectors
large enough for 4, 2 and 1 groups a thread, the last target, odd inner
lengths) and tensors that start between two vectors."""
import numpy as np
import pytest
import torch

from quantumsim_gb300 import _lib as L

pytestmark = pytest.mark.gpu

SHAPES = [((4,) * n, qs) for n, qs in (
    (1, (0,)), (2, (1,)), (2, (0, 1)), (3, (2, 0)), (5, (1, 3)),
    (9, (4,)), (10, (0,)), (10, (9,)), (11, (5,)), (11, (10,)),
    (10, (3, 6)), (11, (0, 5)), (11, (9, 10)), (12, (2, 9)), (12, (11, 10)))]
SHAPES += [((3, 4, 5, 4, 3), (1, 3)), ((3, 4, 4, 6), (1, 2)), ((5, 4, 2), (1,)),
           ((2, 9, 4, 81, 81, 9), (2,)), ((4, 9, 4, 81, 81), (0, 2))]


@pytest.mark.parametrize('shape,qs', SHAPES)
@pytest.mark.parametrize('offset', (0, 1, 2))
def test_full_qubits(shape, qs, offset):
    rng = np.random.default_rng([len(shape), len(qs), offset])
    size = int(np.prod(shape))
    buf = torch.from_numpy(rng.standard_normal(size + offset)).float().cuda()
    x = buf[offset:].view(shape)
    m = rng.standard_normal((4,) * (2 * len(qs)))
    p = torch.from_numpy(m).cuda()
    got = torch.ops.qsgb.apply_ptm(x, p, list(qs), L.ARITH_F32, 0, False)
    k = len(qs)

    def apply(a, b):
        y = torch.tensordot(a, b, dims=(list(range(k, 2 * k)), list(qs)))
        return torch.movedim(y, list(range(k)), list(qs))
    ref = apply(p, x.double())
    # PTM entries rounded to FP32 and one rounding a term: 2^-24 each of the
    # sum of magnitudes, twice the terms at most
    tol = apply(p.abs(), x.double().abs()) * (2 * 4 ** k * 2.0 ** -24)
    assert got.dtype == torch.float32
    assert bool(((got.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize('shape,q,arith', [
    ((4,), 0, L.ARITH_AUTO), ((4, 4), 1, L.ARITH_AUTO),
    ((4,) * 7, 3, L.ARITH_AUTO), ((4,) * 8, 7, L.ARITH_AUTO),
    ((3, 4, 5), 1, L.ARITH_AUTO), ((4,) * 10, 0, L.ARITH_F64),
    ((4,) * 10, 9, L.ARITH_F64), ((7, 4, 4096, 3), 1, L.ARITH_F64)])
@pytest.mark.parametrize('offset', (0, 1))
def test_one_qubit_fp64(shape, q, arith, offset):
    rng = np.random.default_rng([len(shape), q, offset])
    size = int(np.prod(shape))
    buf = torch.from_numpy(rng.standard_normal(size + offset)).cuda()
    x = buf[offset:].view(shape)
    p = torch.from_numpy(rng.standard_normal((4, 4))).cuda()
    got = torch.ops.qsgb.apply_ptm(x, p, [q], arith, 0, False)

    def apply(a, b):
        return torch.movedim(torch.tensordot(a, b, dims=([1], [q])), 0, q)
    # four roundings on either side
    tol = apply(p.abs(), x.abs()) * (8 * 2.0 ** -53)
    assert bool(((got - apply(p, x)).abs() <= tol).all())
