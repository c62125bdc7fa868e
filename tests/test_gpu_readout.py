"""Values read by the host: marginals, diagonal, expectation, partial traces.

The kernels write page-locked host memory themselves; one block or many, by
the number of terms.  Reference: the same sums with numpy in float64.

Tolerance: a value is a sum of N products of n weights and an entry.  Each
product has at most n + 1 roundings and passes at most 64 additions in a thread
plus 32 in shuffles, warps and blocks at these sizes (numpy's pairwise sum:
fewer than 32), so it is within (n + 1 + 64 + 32 + 32) u of the exact sum's
absolute terms, u = 2^-53: below 160 u for n <= 13.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip('torch')

from quantumsim_gb300 import PauliVectorGB300 as GB  # noqa: E402
from quantumsim_gb300 import _lib as L, bases as B, ops  # noqa: E402
from quantumsim_gb300.pauli_vector import _diag_arrays  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 160 * 2.0 ** -53


def make(dims, dtype):
    torch.manual_seed(len(dims))
    s = GB([B.general(d) for d in dims], force=True, dtype=dtype)
    s._data.copy_(torch.randn(s._data.shape, dtype=torch.float64))
    return s, s._data.cpu().numpy().astype(np.float64)


def weighted(x, weights):
    """sum x * prod w over the axes that have weights, and of |terms|."""
    mag = np.abs(x)
    for a in reversed(range(len(weights))):
        if weights[a] is not None:
            w = weights[a].reshape((-1,) + (1,) * (x.ndim - 1 - a))
            x, mag = (x * w).sum(a), (mag * np.abs(w)).sum(a)
    return x, mag


# products of 1, 2, ... terms; 255/256/257 terms a block; odd qudits mixed in
DIMS = [(2,), (3,), (2, 2), (2, 3, 4), (2,) * 6, (3, 2, 3, 2), (2,) * 9,
        (2,) * 11, (5, 3, 5), (17,)]


@pytest.mark.parametrize('dtype', [np.float64, np.float32])
@pytest.mark.parametrize('dims', DIMS, ids=str)
def test_reads(dims, dtype):
    s, x = make(dims, dtype)
    rng = np.random.default_rng(0)
    diag = x[np.ix_(*[range(d) for d in dims])]
    np.testing.assert_array_equal(s.diagonal(), diag.reshape(-1))
    mag = np.abs(diag)
    for _ in range(2):
        assert abs(s.trace() - diag.sum()) <= TOL * mag.sum()
        for q in range(len(dims)):
            rest = tuple(a for a in range(len(dims)) if a != q)
            assert np.all(np.abs(s.meas_prob(q) - diag.sum(rest)) <=
                          TOL * mag.sum(rest))
    for zeros in (False, True):
        ws = [rng.normal(size=d * d) for d in dims]
        if zeros:
            ws[0][1:] = 0
        ref, m = weighted(x, ws)
        got = ops.expectation(s._data, np.concatenate(ws).tolist())
        assert abs(got - ref) <= TOL * m
    assert ops.expectation(s._data, [0.0] * sum(x.shape)) == 0.0


@pytest.mark.parametrize('keep', [(), (0,), (2, 5), (0, 1, 2, 3, 4, 5)])
@pytest.mark.parametrize('dims', [(2,) * 6, (2,) * 8, (2,) * 10], ids=str)
def test_partial_traces(dims, keep):
    """From one output to as many as outputs of one thread each."""
    s, x = make(dims, np.float64)
    flags = [int(a in keep) for a in range(len(dims))]
    ws = [None if f else np.random.default_rng(a).normal(size=4)
          for a, f in enumerate(flags)]
    ref, m = weighted(x, ws)
    flat = [float(v) for w in ws if w is not None for v in w]
    got = torch.ops.qsgb.partial_trace(s._data, flags, flat).cpu().numpy()
    assert np.all(np.abs(got - ref) <= TOL * m)


def test_host_memory_kinds():
    """Page-locked and other host memory get the same values; the gather to
    the host takes page-locked memory alone."""
    s, _ = make((2,) * 9, np.float64)
    arrays = _diag_arrays(s.bases, s._data.shape)
    off, idx, shape, _ = arrays
    dev = torch.empty(8, dtype=torch.float64, device='cuda')
    lib, stream = L.load(), torch.cuda.current_stream().cuda_stream
    want = s.meas_prob(4)
    plain = np.full(8, 7.0)
    assert lib.qsgb_diag_marginals(
        s._data.data_ptr(), L.F64, 9, shape, off, idx, 4, dev.data_ptr(),
        None, plain.ctypes.data, None, 0, stream) == L.OK
    assert np.all(np.abs(plain[:2] - want) <= TOL * np.abs(s.diagonal()).sum())
    np.testing.assert_array_equal(plain[2:], [0.0] + [7.0] * 5)
    np.testing.assert_array_equal(dev.cpu().numpy()[:3], plain[:3])
    big = (ctypes.c_double * 600)()
    assert lib.qsgb_gather_host(s._data.data_ptr(), L.F64, 9, shape, off, idx,
                                None, ctypes.addressof(big),
                                stream) == L.ERR_UNSUPPORTED


def test_status_is_read_along():
    """A device-side status raised earlier on the stream reaches the reader."""
    s, _ = make((2,) * 5, np.float64)
    for read in (s.trace, lambda: s.exp_value('XYZIX'), s.diagonal):
        ops.status_tensor(s.device).fill_(L.DEV_RANGE)
        with pytest.raises(RuntimeError, match='float-float range'):
            read()
        read()


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('shape,idx', [
    ((4,), [[0, 3]]), ((4, 3, 4), [[2], [0, 1, 2], [3, 0]]),
    ((4, 9), [[1, -1], [8, 0, 4]]), ((4,) * 9, [[0, 3]] * 9)], ids=str)
def test_scatter_is_the_adjoint_of_gather(shape, idx, dtype):
    """Whole values: exact."""
    off = np.cumsum([0] + [len(i) for i in idx]).tolist()
    flat = [int(i) for axis in idx for i in axis]
    n = int(np.prod([len(i) for i in idx]))
    g = torch.arange(1, n + 1, dtype=torch.float64, device='cuda')
    got = torch.ops.qsgb.scatter(g, list(shape), off, flat,
                                 dtype == torch.float64)
    assert got.dtype == dtype and got.shape == shape
    ref = np.zeros(shape)
    for o, pos in enumerate(np.ndindex(*[len(i) for i in idx])):
        at = tuple(axis[k] for axis, k in zip(idx, pos))
        if min(at) >= 0:
            ref[at] += o + 1
    np.testing.assert_array_equal(got.cpu().numpy(), ref)
