"""Chains of one kernel whose grids take a fraction, most, all or more than all of
the blocks that the device holds, where launches change between overlapped and
ordinary ones: the same bits as with a synchronisation after every launch."""
import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('where', ['cpu', 'cuda'])
@pytest.mark.parametrize('k', [1, 2])
@pytest.mark.parametrize('blocks', [0.4, 1, 2, 3, 4, 6, 8, 9, 15, 33])
def test_chain(blocks, k, where, dtype):
    rng = np.random.default_rng(int(10 * blocks))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    z = int(blocks * sms * 128) + 2
    m = np.linalg.qr(rng.standard_normal((4 ** k, 4 ** k)))[0]
    if where == 'cpu':
        m = np.where(rng.random(m.shape) < 0.3, m, 0.0) + 0.5 * np.eye(4 ** k)
    p = torch.from_numpy(m.reshape((4,) * (2 * k))).to(where)
    x0 = torch.randn((4,) * k + (z,), device='cuda', dtype=dtype)
    arith = 0 if dtype == torch.float64 else 3

    def run(sync):
        x = x0
        for _ in range(6):
            x = torch.ops.qsgb.apply_ptm(x, p, list(range(k)), arith, 0, False)
            if sync:
                torch.cuda.synchronize()
        return x

    want = run(True)
    for _ in range(3):
        assert torch.equal(run(False), want)
