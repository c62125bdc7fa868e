"""The base-256 digit split of the tensor-core kernels (qsgb_tc.h), modelled in
exact integer arithmetic on the host: digits are FP16 integers built as the
kernel builds them, every level of 16 terms fits the exact range, the pairwise
32-bit and 64-bit recombination neither overflows nor changes the sum, and the
result is as near the exact dot product as the bound says."""
from fractions import Fraction

import numpy as np
import pytest

PLANES, LEVELS = 7, 8
BIAS = 0x0080808080808080


def _split(v, emax):
    """(signed digits, most significant first) of v against emax, as fixed8
    and digit8_pair."""
    b = int(np.float64(v).view(np.uint64))
    hi, lo = b >> 32, b & 0xffffffff
    s = emax - ((hi >> 20) & 0x7ff)
    m = ((((hi & 0xfffff) | 0x100000) << 32) | lo) << 2
    u = ((m >> s) if s < 64 else 0) + BIAS
    assert u >> 56 <= 1  # the top digit carries into bit 56 at most
    out = []
    for j in range(PLANES):
        byte = (u >> (8 * (6 - j))) & (0x1ff if j == 0 else 0xff)
        half = np.array([0x6400 | byte], dtype=np.uint16).view(np.float16)[0]
        d = float(half) - 1152.0
        assert -128 <= d <= 128 and float(np.float16(d)) == d
        out.append(int(-d if b >> 63 else d))
    return out


def _emax(v):
    e = (np.abs(v).view(np.uint64) >> np.uint64(52)).astype(int).max()
    return int(e) if e >= 64 else 1023


def _i32(x):
    assert -2 ** 31 <= x < 2 ** 31
    return x


def _dot(p, x):
    ep, ex = _emax(p), _emax(x)
    pd, xd = [_split(v, ep) for v in p], [_split(v, ex) for v in x]
    lev = []
    for L in range(LEVELS):
        a = sum(pd[k][i] * xd[k][L - i] for k in range(len(x))
                for i in range(max(0, L - 6), min(6, L) + 1))
        assert abs(a) < 1 << 22  # exact in FP32, and with 1.5 * 2^23 added
        lev.append(a)
    q = [_i32(256 * lev[2 * i] + lev[2 * i + 1]) for i in range(4)]
    v = (q[1] << 18) + _i32(q[2] * 4 + (q[3] >> 14)) + (q[0] << 34)
    assert abs(v) < 1 << 61
    return Fraction(v) * Fraction(2) ** (ex + ep - 2100)


def _vectors(kind, rng):
    if kind == 'ones':  # the largest digits and level sums
        top = np.nextafter(2.0, 0.0)
        return np.full(16, top), np.full(16, -top)
    if kind == 'alternating':
        return np.tile([1.0, -1.0], 8) * 1.9375, np.full(16, 1.00390625)
    if kind == 'zeros':
        p, x = rng.standard_normal(16), np.zeros(16)
        x[3] = -0.0
        return p, x
    spread = {'flat': 0.0, 'wide': 3.0, 'sparse': 1.0}[kind]
    p = rng.standard_normal(16) * np.exp(rng.normal(0, spread, 16))
    x = rng.standard_normal(16) * np.exp(rng.normal(0, spread, 16))
    if kind == 'sparse':
        x[rng.random(16) < 0.6] = 0.0
        p[rng.random(16) < 0.4] = 0.0
        x[5], p[5] = 1.0, 1.0
    return p, x


@pytest.mark.parametrize('kind', ['ones', 'alternating', 'zeros', 'flat',
                                  'wide', 'sparse'])
def test_split_and_recombination(kind):
    rng = np.random.default_rng(3)
    for _ in range(40):
        p, x = _vectors(kind, rng)
        exact = sum(Fraction(float(a)) * Fraction(float(b))
                    for a, b in zip(p, x))
        scale = Fraction(float(np.abs(p).max())) * \
            Fraction(float(np.abs(x).max()))
        # dropped levels 5 pairs * 2^14 * 2^(8 * 4) of 2^108 a term, truncation
        # 2^-55 of each factor, the last 2 of the recombined units
        bound = (16 * (5 * Fraction(2) ** (14 + 32 + 1 - 108) * 4 +
                       2 * Fraction(2) ** -54) +
                 2 * Fraction(2) ** -54) * scale
        assert abs(_dot(p, x) - exact) <= bound
