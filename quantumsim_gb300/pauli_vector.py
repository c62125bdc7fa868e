"""``PauliVectorGB300``: the GB300 density-matrix backend.

A drop-in ``PauliVectorBase`` subclass with the surface of the reference
backends (quantumsim/pauli_vectors/numpy.py:8-121 and
quantumsim/pauli_vectors/cuda.py:55-425): ``apply_ptm`` for one and two
qudits on any indices (rectangular PTMs included), ``diagonal``,
``meas_prob``, ``trace``, ``partial_trace``, ``renormalize`` and ``copy``,
plus ``reduce_basis`` and ``project``.  All device work goes through the
``torch.ops.qsgb`` operators over ``libqsgb.so``; there is no CPU path.

Numerical semantics follow ``PauliVectorNumpy`` (the reference oracle):

* the initial state puts 1 at index (0, ..., 0) (numpy.py:39-41);
* ``diagonal()`` has length prod(dim_hilbert) and contracts each qudit with
  ``computational_basis_vectors`` (numpy.py:66-80); for bases whose rows are
  unit vectors (``general(d)`` and its subbases) that is an exact gather;
* ``meas_prob`` returns an ndarray of length d_hilbert (numpy.py:97-107);
* ``partial_trace(*qubits)`` keeps ``qubits``: data axes in ascending qudit
  order, ``bases`` in argument order (numpy.py:86-95);
* ``renormalize`` warns when the trace is <= 1e-8 and returns the trace
  before scaling (numpy.py:109-117).

FP64 storage: by default (``arith='auto'``) the kernel computes each PTM
row either with native FP64 FMAs or in float-float arithmetic (48-bit
significand) on the FP32 pipes, whichever keeps the launch closest to the
HBM bound, and sends dense PTMs (16 x 16 with more than 8 non-zero terms per
row; larger ones without zeros) to the tensor cores, where FP64 values split
into FP16 digit planes are multiplied with exact FP32 sums.  The digits are cut
at 55 bits below the largest input of a group, so components far below it keep
fewer bits of their own there.  ``arith='f64'`` forces native FP64
everywhere, ``arith='df64'`` float-float for every row with more than one
term (both keep every component's own precision), and ``arith='tc'`` the
tensor cores for every 16 x 16 PTM.
``dtype=np.float32`` stores the vector in FP32 while every trace, marginal
and partial-trace sum still accumulates in FP64.
"""
import collections
import hashlib
import math
import warnings

import numpy as np
import torch

from . import _lib as L
from . import ops

# Pauli matrices of the operator strings of exp_value
# (quantumsim/algebra/tools.py:4-13)
_PAULI = {
    'I': np.array([[1, 0], [0, 1]], dtype=complex),
    'X': np.array([[0, 1], [1, 0]], dtype=complex),
    'Y': np.array([[0, -1j], [1j, 0]], dtype=complex),
    'Z': np.array([[1, 0], [0, -1]], dtype=complex),
}

try:  # subclass the reference ABC when the quantumsim package is present
    with warnings.catch_warnings():
        warnings.simplefilter('ignore')
        from quantumsim.pauli_vectors.pauli_vector import \
            PauliVectorBase as _Base
    REFERENCE_BASE = True
except Exception:  # pragma: no cover - depends on the environment
    from ._base import PauliVectorBase as _Base
    REFERENCE_BASE = False

_ARITH = {'auto': L.ARITH_AUTO, 'df64': L.ARITH_DF64, 'f64': L.ARITH_F64,
          'f32': L.ARITH_F32, 'tc': L.ARITH_TC}


class _PtmCache:
    """Device copies of PTMs too large to travel in a kernel launch, keyed
    by content (the reference keys on hash(bytes), cuda.py:401-420), LRU."""

    def __init__(self, capacity=1024):
        self.capacity = capacity
        self._d = collections.OrderedDict()

    def get(self, ptm, device):
        key = (hashlib.blake2b(ptm.tobytes(), digest_size=16).digest(),
               ptm.shape, str(device))
        t = self._d.get(key)
        if t is None:
            t = torch.from_numpy(ptm).to(device)
            self._d[key] = t
            if len(self._d) > self.capacity:
                self._d.popitem(last=False)
        else:
            self._d.move_to_end(key)
        return t


_PTM_CACHE = _PtmCache()

# validated plans of eager host-PTM applications (see ops.eager_plan)
_APPLY_PLANS = {}


_PLAN_CACHE = {}


def _diag_plan(bases):
    """Gather plan for diagonal(): per qudit, for each Hilbert index i the
    Pauli index x whose computational_basis_vectors row is exactly e_x, or
    -1 for an all-zero row.  None if some row is neither.  Cached by the
    identity of the basis objects (the cache keeps them alive, so an id is
    never reused while its entry exists)."""
    key = tuple(id(b) for b in bases)
    hit = _PLAN_CACHE.get(key)
    if hit is not None:
        return hit[1]
    plan = _diag_plan_of(bases)
    if len(_PLAN_CACHE) > 256:
        _PLAN_CACHE.clear()
    _PLAN_CACHE[key] = (tuple(bases), plan)
    return plan


_DIAG_ARRAYS = {}


def _diag_arrays(bases, shape):
    """The gather plan of _diag_plan as C arrays for ops.diag_marginals
    (index offsets, indices, vector shape, outcomes per qudit), or None for
    bases without a gather plan.  Cached like _diag_plan."""
    key = (tuple(id(b) for b in bases), tuple(shape))
    hit = _DIAG_ARRAYS.get(key)
    if hit is not None:
        return hit[1]
    plan = _diag_plan(bases)
    arrays = None
    if plan is not None:
        idx_off, idx = plan
        arrays = (L.i32_array(idx_off), L.i32_array(idx), L.i64_array(shape),
                  [idx_off[a + 1] - idx_off[a] for a in range(len(bases))])
    if len(_DIAG_ARRAYS) > 256:
        _DIAG_ARRAYS.clear()
    _DIAG_ARRAYS[key] = (tuple(bases), arrays)
    return arrays


def _diag_plan_of(bases):
    idx_off, idx = [0], []
    for b in bases:
        cbv = np.asarray(b.computational_basis_vectors)
        if np.any(np.imag(cbv) != 0):
            return None
        cbv = np.real(cbv)
        for row in cbv:
            nz = np.flatnonzero(row)
            if len(nz) == 0:
                idx.append(-1)
            elif len(nz) == 1 and row[nz[0]] == 1.0:
                idx.append(int(nz[0]))
            else:
                return None
        idx_off.append(len(idx))
    return idx_off, idx


class PauliVectorGB300(_Base):
    """Density matrix in a Pauli basis, stored on a GB300 (CUDA) device.

    Parameters
    ----------
    bases : list of PauliBasis
        Basis of every qudit.
    pv : numpy array, torch tensor or None
        Expansion coefficients, shape ``dim_pauli``; None = |0...0><0...0|
        (coefficient 1 at index (0, ..., 0)).
    force : bool
        Allow more than 2**22 density-matrix elements.
    dtype : np.float64 (default) or np.float32
        Storage type of the Pauli vector on the device.
    device : torch device or None
        CUDA device (default: the current one).
    arith : 'auto' | 'df64' | 'f64' | 'f32' | 'tc'
        Arithmetic of apply_ptm ('auto': per PTM, the specialised
        float-float / FP64 kernels, or the tensor cores for dense PTMs, see
        above; 'tc': every 16 x 16 PTM on the
        tensor cores; f32 for FP32 storage).
    """

    def __init__(self, bases, pv=None, *, force=False, dtype=None,
                 device=None, arith='auto'):
        super().__init__(bases, pv, force=force)
        if not torch.cuda.is_available():
            raise RuntimeError('PauliVectorGB300 needs a CUDA device')
        self._device = torch.device(device) if device is not None else \
            torch.device('cuda', torch.cuda.current_device())
        if self._device.type != 'cuda':
            raise ValueError('PauliVectorGB300 lives on a CUDA device')
        if dtype is None:
            tdtype = (pv.dtype if isinstance(pv, torch.Tensor) and
                      pv.dtype == torch.float32 else torch.float64)
        else:
            tdtype = torch.float32 if np.dtype(dtype) == np.float32 else \
                torch.float64
            if np.dtype(dtype) not in (np.float32, np.float64):
                raise ValueError('dtype must be float64 or float32')
        if arith not in _ARITH:
            raise ValueError('arith must be one of {}'.format(list(_ARITH)))
        if arith == 'f32' and tdtype != torch.float32 or \
                arith in ('df64', 'f64', 'tc') and tdtype != torch.float64:
            raise ValueError('arith {!r} does not match storage {}'.format(
                arith, tdtype))
        if arith == 'auto' and tdtype == torch.float32:
            arith = 'f32'
        self._arith_key = arith
        self._arith = _ARITH[arith]

        if pv is None:
            data = torch.zeros(self.dim_pauli, dtype=tdtype,
                               device=self._device)
            data[(0,) * self.n_qubits] = 1
        elif isinstance(pv, np.ndarray):
            if pv.shape != self.dim_pauli:
                raise ValueError(
                    '`bases` Pauli dimensionality should be the same as the '
                    'shape of `data` array.\n - bases shapes: {}\n - data '
                    'shape: {}'.format(self.dim_pauli, pv.shape))
            if pv.dtype not in (np.float16, np.float32, np.float64):
                raise ValueError('`pv` must have floating point data type, '
                                 'got {}'.format(pv.dtype))
            data = torch.from_numpy(np.ascontiguousarray(pv)).to(
                device=self._device, dtype=tdtype)
        elif isinstance(pv, torch.Tensor):
            if tuple(pv.shape) != self.dim_pauli:
                raise ValueError(
                    '`bases` Pauli dimensionality should be the same as the '
                    'shape of `data` array.\n - bases shapes: {}\n - data '
                    'shape: {}'.format(self.dim_pauli, tuple(pv.shape)))
            if pv.dtype not in (torch.float16, torch.float32, torch.float64):
                raise ValueError('`pv` must have floating point data type, '
                                 'got {}'.format(pv.dtype))
            # (the kernels read its memory: no lazily negated view)
            data = pv.to(device=self._device,
                         dtype=tdtype).contiguous().resolve_neg()
        else:
            raise ValueError('`pv` should be a numpy array, a torch tensor or '
                             'None, got type `{}`'.format(type(pv)))
        self._data = data
        # the state buffer of two applications back, written by the next
        # apply_ptm instead of a new tensor (the reference swaps two
        # buffers the same way, cuda.py:113-115, 221); only tensors this
        # object allocated and never handed out take that role
        self._owned = False
        self._work = None

    # ------------------------------------------------------------ accessors
    @property
    def data(self):
        """The device tensor (shape ``dim_pauli``).  A tensor handed out
        here is never reused as a work buffer: later operations leave it
        as it is."""
        self._owned = False
        return self._data

    @property
    def device(self):
        return self._device

    @property
    def dtype(self):
        return np.float64 if self._data.dtype == torch.float64 else np.float32

    def to_pv(self):
        ops.check_device_status(self._device)
        return self._data.cpu().numpy()

    def copy(self):
        return self.__class__(self.bases, self._data.clone(), force=True,
                              dtype=self.dtype, device=self._device,
                              arith=self._arith_name())

    def _arith_name(self):
        return self._arith_key

    # ------------------------------------------------------------ apply_ptm
    def _device_ptm(self, ptm):
        """PTMs stay on the host: the library reads them during the call
        (their sparsity pattern picks a kernel specialised at run time) and
        passes the values inside the kernel launch."""
        return torch.from_numpy(ptm)

    def apply_ptm(self, ptm, *qubits):
        """Apply a PTM of shape (d_out..., d_in...) to `qubits` (argument
        order, any position); ``bases`` are left to the caller
        (quantumsim/operations/operation.py:549-551)."""
        if type(ptm) is np.ndarray:
            # host PTM: a validated plan per geometry, then one C call
            # (which takes any float64 layout and dtype, converting when needed)
            data = self._data
            key = (data.shape, data.dtype, qubits, ptm.shape)
            plan = _APPLY_PLANS.get(key)
            if plan is None:
                self._validate_apply(ptm.shape, qubits)
                plan = ops.eager_plan(tuple(data.shape), data.dtype, qubits,
                                      ptm.shape)
                if len(_APPLY_PLANS) > 4096:
                    _APPLY_PLANS.clear()
                _APPLY_PLANS[key] = plan
            work = self._work
            if work is not None and work.shape != plan[0]:
                self._work = work = None
            out = None
            if ptm.size > ops.MAX_JIT_TERMS:
                out = ops.eager_apply_dense(data, ptm, plan, self._arith,
                                            work)
            if out is None:
                out = ops.eager_apply(data, ptm, plan, self._arith, work)
            if out is not None:
                self._work = data if self._owned else None
                self._data = out
                self._owned = True
                return
        self._apply_general(ptm, *qubits)

    def _validate_apply(self, shape, qubits):
        """The reference's argument errors for a PTM of `shape` on
        `qubits` (quantumsim/pauli_vectors/pauli_vector.py:102-116,
        cuda.py:125-127, 164-168, 240-243)."""
        n = len(qubits)
        if len(shape) != 2 * n:
            raise ValueError('{}-qubit PTM must have {} dimensions, got {}'
                             .format(n, 2 * n, len(shape)))
        if n == 0:
            raise NotImplementedError('Applying a 0-qubit PTM is not '
                                      'implemented in this backend.')
        if n > 2:
            raise NotImplementedError('Applying {}-qubit PTM is not '
                                      'implemented in the active backend.'
                                      .format(n))
        for i, q in enumerate(qubits):
            self._validate_qubit(q, 'qubit{}'.format(i))
        if n == 2 and qubits[0] == qubits[1]:
            raise ValueError('The two qubits of a 2-qubit PTM must differ')
        for q, din in zip(qubits, shape[n:]):
            if self._data.shape[q] != din:
                raise ValueError(
                    'PTM acts on a {}-dimensional Pauli space, qubit {} has '
                    'dim_pauli {}'.format(din, q, self._data.shape[q]))

    def _apply_general(self, ptm, *qubits):
        n = len(qubits)
        if isinstance(ptm, torch.Tensor):
            ptm_t = ptm.to(torch.float64)
            shape = tuple(ptm_t.shape)
        else:
            ptm = np.ascontiguousarray(ptm, dtype=np.float64)
            shape = ptm.shape
            ptm_t = None
        if len(shape) != 2 * n:
            raise ValueError('{}-qubit PTM must have {} dimensions, got {}'
                             .format(n, 2 * n, len(shape)))
        if n == 0:
            raise NotImplementedError('Applying a 0-qubit PTM is not '
                                      'implemented in this backend.')
        if n > 2:
            raise NotImplementedError('Applying {}-qubit PTM is not '
                                      'implemented in the active backend.'
                                      .format(n))
        for i, q in enumerate(qubits):
            self._validate_qubit(q, 'qubit{}'.format(i))
        if n == 2 and qubits[0] == qubits[1]:
            raise ValueError('The two qubits of a 2-qubit PTM must differ')
        for q, din in zip(qubits, shape[n:]):
            if self._data.shape[q] != din:
                raise ValueError(
                    'PTM acts on a {}-dimensional Pauli space, qubit {} has '
                    'dim_pauli {}'.format(din, q, self._data.shape[q]))
        if ptm_t is None:
            max_terms = 0  # host PTM: the library counts its terms
            ptm_t = self._device_ptm(ptm)
        else:
            max_terms = 0 if not ptm_t.is_cuda else math.prod(shape)
        self._data = torch.ops.qsgb.apply_ptm(
            self._data, ptm_t, list(qubits), self._arith, max_terms, False)

    # ------------------------------------------------------------ diagonal
    def _diagonal_device(self):
        """FP64 device tensor of length prod(dim_hilbert)."""
        plan = _diag_plan(self.bases)
        if self.n_qubits == 0:
            return self._data.reshape(1).to(torch.float64, copy=True)
        if plan is not None:
            idx_off, idx = plan
            return torch.ops.qsgb.gather(self._data, idx_off, idx, True)
        # general bases: contract each qudit with its (real) computational
        # basis vectors, d_hilbert x d_pauli, as a rectangular 1-qudit PTM
        data = self._data if self._data.dtype == torch.float64 else \
            self._data.to(torch.float64)
        for q, b in enumerate(self.bases):
            m = np.ascontiguousarray(
                np.real(b.computational_basis_vectors), dtype=np.float64)
            data = torch.ops.qsgb.apply_ptm(
                data, self._device_ptm(m), [q], L.ARITH_DF64,
                ops.nnz_terms(m, L.ARITH_DF64), False)
        return data.reshape(-1)

    def diagonal(self, *, get_data=True, target_array=None, flatten=True):
        """Probabilities of the computational basis states, length
        prod(dim_hilbert) (quantumsim/pauli_vectors/numpy.py:66-80).
        `get_data=False` returns the float64 CUDA tensor.  As in the
        reference's GPU backend (quantumsim/pauli_vectors/cuda.py:279-345),
        `target_array` is an already allocated CUDA tensor that receives the
        values (ValueError when too small), and `flatten=False` shapes the
        result as dim_hilbert."""
        if get_data and target_array is None and \
                not self._data.requires_grad and self._data.is_contiguous():
            arrays = _diag_arrays(self.bases, self._data.shape)
            if arrays is not None:
                out = ops.diagonal_host(self._data, arrays)
                if out is not None:
                    return out if flatten else out.reshape(
                        tuple(self.dim_hilbert))
        diag = self._diagonal_device()
        if target_array is not None:
            n = diag.numel()
            if target_array.numel() < n:
                raise ValueError(
                    'Size of `target_array` is too small ({}).\n'
                    'Should be at least {}.'.format(target_array.numel(), n))
            view = target_array.reshape(-1)[:n]
            view.copy_(diag)
            diag = view
        if not get_data:
            return diag if flatten else diag.reshape(tuple(self.dim_hilbert))
        out = ops.fetch_checked(diag)
        return out if flatten else out.reshape(tuple(self.dim_hilbert))

    def _trace_device(self):
        diag = self._diagonal_device()
        return torch.ops.qsgb.marginals(diag, [diag.numel()], -1)

    def _diag_reduce(self, axis):
        """Trace (axis -1) or marginals of one qudit in one launch, which
        writes them to the host (ops.diag_marginals); None when the bases have no
        gather plan or the diagonal is too large for the fused kernel."""
        arrays = _diag_arrays(self.bases, self._data.shape)
        if arrays is None:
            return None
        return ops.diag_marginals(self._data, arrays, axis)

    def trace(self):
        vals = self._diag_reduce(-1)
        if vals is not None:
            return float(vals[0])
        return float(ops.fetch_checked(self._trace_device())[0])

    def meas_prob(self, qubit):
        self._validate_qubit(qubit, 'qubit')
        vals = self._diag_reduce(qubit)
        if vals is not None:
            return vals
        diag = self._diagonal_device()
        probs = torch.ops.qsgb.marginals(diag, list(self.dim_hilbert), qubit)
        return ops.fetch_checked(probs)

    def partial_trace(self, *qubits):
        for q in qubits:
            self._validate_qubit(q, 'qubit')
        keep = [1 if i in qubits else 0 for i in range(self.n_qubits)]
        weights = []
        for i, b in enumerate(self.bases):
            if not keep[i]:
                weights.extend(float(w) for w in
                               np.real(np.einsum('xkk->x', b.vectors)))
        data = torch.ops.qsgb.partial_trace(self._data, keep, weights)
        return self.__class__([self.bases[q] for q in qubits], data,
                              force=True, dtype=self.dtype,
                              device=self._device, arith=self._arith_name())

    def renormalize(self):
        tr = self.trace()
        if tr > 1e-8:
            torch.ops.qsgb.scale_(self._data, 1.0 / tr)
        else:
            warnings.warn(
                'Density matrix trace is 0; likely your further computation '
                'will fail. Have you projected DM on a state with zero '
                'weight?')
        return tr

    # ------------------------------------------------------------ new API
    def exp_value(self, operator):
        """Expectation value tr(rho O) of a Pauli string `operator` (one of
        I, X, Y, Z per qubit, any case), computed on the device.

        The reference contracts the host copy of the Pauli vector with
        sigma_q[a, b] and each basis' vectors[k, b, a]
        (quantumsim/states/state.py:43-83).  For a string that contraction is
        sum_k pv[k] prod_q w_q[k_q] with w_q[k] = tr(sigma_q P_k): the
        weighted full contraction of the partial-trace kernel with no qudit
        kept (FP64 accumulation).  Same ValueErrors as the reference; the
        value is returned as a float (the reference's einsum returns the
        same number as a complex with zero imaginary part).  Dense operator
        arrays are left to the reference's host contraction."""
        if not isinstance(operator, str):
            raise NotImplementedError(
                'exp_value on the device takes Pauli strings; dense operators '
                'are contracted on the host by State.exp_value')
        n = self.n_qubits
        if n != len(operator):
            raise ValueError("operator string must have the same length "
                             "as number of qubits in the state")
        try:
            sigmas = [_PAULI[ch.upper()] for ch in operator]
        except KeyError as ex:
            raise ValueError("operator string must contain only I, X, "
                             "Y or Z") from ex
        weights = []
        for s, b in zip(sigmas, self.bases):
            if b.dim_hilbert != 2:
                raise ValueError('Pauli strings act on qubits; qudit basis '
                                 'of dimension {}'.format(b.dim_hilbert))
            w = np.einsum('ab,kba->k', s, np.asarray(b.vectors))
            weights.extend(float(v) for v in np.real(w))
        if not self._data.requires_grad:
            return ops.expectation(self._data, weights)
        out = torch.ops.qsgb.partial_trace(self._data, [0] * n, weights)
        return float(ops.fetch_checked(out)[0])

    def reduce_basis(self, qubit, indices):
        """Keep only the Pauli elements `indices` of `qubit`'s basis
        (e.g. 9 -> 3 with the computational subbasis of a qutrit) and
        switch its basis to ``bases[qubit].subbasis(indices)``.  Same result
        as ``apply_ptm(np.eye(d)[indices], qubit)`` followed by the basis
        update of quantumsim/operations/operation.py:549-551."""
        self._validate_qubit(qubit, 'qubit')
        indices = [int(i) for i in indices]
        d = self._data.shape[qubit]
        if not indices or any(i < 0 or i >= d for i in indices):
            raise ValueError('basis indices must be within [0, {})'.format(d))
        self._data = torch.ops.qsgb.take_axis(self._data, qubit, indices)
        self._work = None
        self.bases[qubit] = self.bases[qubit].subbasis(indices)

    def project(self, qubit, state):
        """Project `qubit` onto computational state `state` (its basis shrinks
        to the single element |state><state|).  The trace afterwards is the
        outcome's probability; call :meth:`renormalize` to normalise."""
        self._validate_qubit(qubit, 'qubit')
        idx = self.bases[qubit].computational_basis_indices.get(state)
        if idx is None:
            raise ValueError('state {} of qubit {} has no computational '
                             'basis element in its basis'.format(state, qubit))
        self.reduce_basis(qubit, [idx])


def register(make_default=False):
    """Expose the backend as ``quantumsim.pauli_vectors.PauliVectorGB300``
    (and module ``quantumsim.pauli_vectors.gb300``) when quantumsim is
    importable.  Returns True if registered."""
    import sys
    try:
        with warnings.catch_warnings():
            warnings.simplefilter('ignore')
            import quantumsim.pauli_vectors as qpv
    except Exception:
        return False
    qpv.PauliVectorGB300 = PauliVectorGB300
    if 'PauliVectorGB300' not in qpv.__all__:
        qpv.__all__.append('PauliVectorGB300')
    sys.modules.setdefault('quantumsim.pauli_vectors.gb300',
                           sys.modules[__name__])
    if make_default:
        qpv.Default = PauliVectorGB300
    return True
