"""16 x 16 PTM gradients on the tensor cores: chunks of 16 and of 32 groups.

Above the number of resident warps the chunks have 32 groups; at the last qudit
a group's rows are read as 32-byte words when the tensors are aligned to them.

Tolerance: a chunk's digit products beyond the kept levels are below
2^-49 max|g| max|x| for 16 groups (twice that for 32, half as many chunks), and
the FP64 sums over chunks, warps and blocks round at 2^-53 of partial sums of
at most 16 max|g| max|x| per chunk, fewer than 64 times each:
chunks16 (2^-49 + 64 * 16 * 2^-53) max|g| max|x|.  The numpy reference (pairwise
sums) is far inside.
"""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

import quantumsim_gb300  # noqa: E402,F401

pytestmark = pytest.mark.gpu


def limit():
    """Groups up to which the chunks have 16."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return sms * 2 * 8 * 16


def check(x, g, qs):
    got = torch.ops.qsgb.ptm_grad(x, g, list(qs)).reshape(16, 16).cpu().numpy()
    xs, gs = (np.moveaxis(t.cpu().numpy(), qs, (0, 1)).reshape(16, -1)
              for t in (x, g))
    with np.errstate(invalid='ignore'):
        ref = np.stack([(gs[r] * xs).sum(-1) for r in range(16)])
    chunks = -(-xs.shape[1] // 16)
    fx, fg = (np.where(np.isfinite(v), v, 0) for v in (xs, gs))
    tol = chunks * (2.0 ** -49 + 1024 * 2.0 ** -53) * np.abs(fx).max() * \
        np.abs(fg).max()
    fin = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(got), fin)
    assert np.all(np.abs(got[fin] - ref[fin]) <= tol)
    return got


@pytest.mark.parametrize('extra', [-1, 0, 1, 15, 17, 33, 4000])
@pytest.mark.parametrize('place', ['first', 'last', 'around'])
def test_chunk_sizes(extra, place):
    n = limit() + extra
    torch.manual_seed(n)
    shape, qs = {'first': ((4, 4, n), (0, 1)), 'last': ((n, 4, 4), (1, 2)),
                 'around': ((4, n, 4), (2, 0))}[place]
    x, g = (torch.randn(shape, dtype=torch.float64, device='cuda')
            for _ in range(2))
    got = check(x, g, qs)
    # the same values off the 32-byte boundary: the same bits
    def shifted(t):
        buf = torch.empty(t.numel() + 1, dtype=t.dtype, device='cuda')
        return buf[1:].view(t.shape).copy_(t)
    off = torch.ops.qsgb.ptm_grad(shifted(x), shifted(g), list(qs))
    np.testing.assert_array_equal(off.reshape(16, 16).cpu().numpy(), got)


@pytest.mark.parametrize('value', [0.0, 1e-305, 1e300, np.inf, np.nan])
def test_values_without_digits(value):
    """Chunks of 32 that the digits cannot hold are computed in FP64."""
    n = limit() + 5
    torch.manual_seed(1)
    x, g = (torch.randn((n, 4, 4), dtype=torch.float64, device='cuda')
            for _ in range(2))
    x[n // 2:n // 2 + 40, 1, 2] = value
    g[:, 3, 3] = 0.0
    check(x, g, (1, 2))


@pytest.mark.parametrize('n', [1, 15, 300, 'limit', 'above'])
@pytest.mark.parametrize('place', ['first', 'last'])
@pytest.mark.parametrize('value', [1.0, 0.0, 1e-40, 3e38, np.inf, np.nan])
def test_fp32_vectors(n, place, value):
    """FP32 values are split as they are; subnormals go to FP64."""
    n = {'limit': limit(), 'above': limit() + 21}.get(n, n)
    torch.manual_seed(n)
    shape, qs = {'first': ((4, 4, n), (0, 1)),
                 'last': ((n, 4, 4), (1, 2))}[place]
    x, g = (torch.randn(shape, dtype=torch.float64, device='cuda').float()
            for _ in range(2))
    x[n // 2 if place == 'last' else 1] *= float(np.float32(value))
    got = torch.ops.qsgb.ptm_grad(x, g, list(qs)).cpu()
    check(x.double(), g.double(), qs)  # the FP64 kernel on the same values
    xs, gs = (np.moveaxis(t.double().cpu().numpy(), qs, (0, 1))
              .reshape(16, -1) for t in (x, g))
    with np.errstate(invalid='ignore', over='ignore'):
        ref = np.stack([(gs[r] * xs).sum(-1) for r in range(16)])
    fin = np.isfinite(ref)
    got = got.reshape(16, 16).numpy()
    np.testing.assert_array_equal(np.isfinite(got), fin)
    fx, fg = (np.where(np.isfinite(v), np.abs(v), 0) for v in (xs, gs))
    tol = -(-n // 16) * (2.0 ** -49 + 1024 * 2.0 ** -53) * fx.max() * fg.max()
    assert np.all(np.abs(got[fin] - ref[fin]) <= tol)
