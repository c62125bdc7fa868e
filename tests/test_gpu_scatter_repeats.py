"""scatter with an index named more than once: the values that meet in an
element are added in FP64, in a fixed order, and stored once."""
import numpy as np
import pytest
import torch

import quantumsim_gb300  # noqa: F401  (registers the operators)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('shape,idx', [
    ((4,), [[2] * 700]), ((4, 3), [[1, 1, 0] * 20, [2, 2]]),
    ((4, 4, 4), [[0] * 9, [3, -1, 3], [1, 2] * 8]),
    ((9, 4) + (4,) * 5, [[8, 8], [0, 3, 3]] + [[0, 3]] * 5)], ids=str)
def test_repeated_indices(shape, idx, dtype):
    off = np.cumsum([0] + [len(i) for i in idx]).tolist()
    flat = [int(i) for axis in idx for i in axis]
    n = int(np.prod([len(i) for i in idx]))
    # one large value among many whose FP32 sum with it would lose them
    v = np.full(n, 2.0 ** -25)
    v[n // 2] = 1.0
    v[::3] *= -0.5
    g = torch.from_numpy(v).cuda()
    runs = [torch.ops.qsgb.scatter(g, list(shape), off, flat,
                                   dtype == torch.float64).cpu()
            for _ in range(3)]
    ref = np.zeros(shape)
    for o, pos in enumerate(np.ndindex(*[len(i) for i in idx])):
        at = tuple(axis[k] for axis, k in zip(idx, pos))
        if min(at) >= 0:
            ref[at] += v[o]  # exact: multiples of 2^-26 below 2
    for got in runs:
        want = ref.astype(np.float32 if dtype == torch.float32 else
                          np.float64)
        assert int((got.numpy() != want).sum()) == 0
