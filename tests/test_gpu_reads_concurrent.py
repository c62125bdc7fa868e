"""Values read by several threads and on several streams at a time: each gets
its own state's, to the bit, again and again."""
import threading

import numpy as np
import pytest
import torch

import quantumsim_gb300 as qg
from quantumsim_gb300 import bases as B

pytestmark = pytest.mark.gpu


def _reads(pv, n, string):
    out = [pv.trace(), pv.exp_value(string)]
    out += [pv.meas_prob(q) for q in range(n)]
    return out + [pv.diagonal()]


@pytest.mark.parametrize('n', [4, 11])
@pytest.mark.parametrize('threads,streams', [(1, 2), (2, 1), (4, 4)])
def test_concurrent_reads(n, threads, streams):
    count = max(threads, streams)
    pvs, want = [], []
    string = ''.join('IXYZ'[i % 4] for i in range(n))
    for i in range(count):
        x = np.random.default_rng(i).standard_normal((4,) * n)
        pvs.append(qg.PauliVectorGB300([B.general(2)] * n, x, force=True))
        want.append(_reads(pvs[i], n, string))
    torch.cuda.synchronize()
    sts = [torch.cuda.Stream() for _ in range(streams)]
    bad = []

    def work(t):
        try:
            for rep in range(20):
                for i in range(t, count, threads):
                    with torch.cuda.stream(sts[(i + rep) % streams]):
                        got = _reads(pvs[i], n, string)
                    for a, b in zip(got, want[i]):
                        if not np.array_equal(a, b):
                            bad.append((t, rep, i))
        except Exception as e:
            bad.append(e)

    pool = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not bad


def test_gradients_in_threads():
    """Host PTM gradients on two threads: each its own memory and event."""
    rng = np.random.default_rng(5)
    p = [torch.from_numpy(rng.normal(size=(4,) * 4)) for _ in range(2)]
    x = torch.from_numpy(rng.normal(size=(4,) * 6)).cuda()

    def grads(i):
        a, q = x.clone().requires_grad_(True), p[i].clone().requires_grad_()
        y = qg.apply_ptm_diff(qg.apply_ptm_diff(a, q, i, 4), q, 5, 2 + i)
        return torch.autograd.grad((y * y).sum(), (a, q))

    want = [grads(i) for i in range(2)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got = grads(i)
                torch.cuda.current_stream().synchronize()
                if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                    bad.append(i)

    pool = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not bad


@pytest.mark.parametrize('n,axis', [(3, -1), (9, 4), (12, -1)])
def test_device_results_are_complete_on_return(n, axis):
    """The call returns on a flag that the kernel writes, not when the stream is
    idle: the results on the device, the status among them, are there by then
    for work on any other stream, and the scratch is free."""
    from quantumsim_gb300 import _lib as L
    from quantumsim_gb300.pauli_vector import _diag_arrays
    pv = qg.PauliVectorGB300([B.general(2)] * n, force=True)
    off, idx, shape, _ = _diag_arrays(pv.bases, pv._data.shape)
    lib = L.load()
    count = 1 if axis < 0 else 2
    dev = torch.empty(4, dtype=torch.float64, device='cuda')
    host = torch.empty(4, dtype=torch.float64, pin_memory=True)
    status = torch.tensor([3], dtype=torch.int32, device='cuda')
    nscr = int(lib.qsgb_diag_marginals_scratch_bytes())
    scratch = torch.zeros(nscr, dtype=torch.uint8, device='cuda')
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    want = [1.0, 3.0] if axis < 0 else [1.0, 0.0, 3.0]
    for i in range(200):
        dev.fill_(-1.0)
        torch.cuda.synchronize()
        st = lib.qsgb_diag_marginals(
            pv._data.data_ptr(), L.F64, n, shape, off, idx, axis,
            dev.data_ptr(), status.data_ptr(), host.data_ptr(),
            scratch.data_ptr(), nscr, (a, b)[i % 2].cuda_stream)
        with torch.cuda.stream((b, a)[i % 2]):
            got = dev[:count + 1].cpu().tolist()
        assert st == L.OK and got == want and host[:count + 1].tolist() == want
