"""Sums of the largest digits.  Fields whose leading six digits are 250 to 255 of at
most 256 (at random: sums of equal ones would end in zeros), against matrices whose
entries barely change along the sum and have 255 in their leading three: the sums of
groups 0 to 3 come within a few percent of the 2^24 that an FP32 accumulator holds
exactly.  A run that drained one chain too late would lose units of its group, 1e-10
of a result and more.

The field changes along its columns only, so that F[u][v] = S1[u] S2[v] with S1 the
sums of its values and matrix entries, S2 those of matrix entries, from phases taken
in rationals.  Bound: an entry's error of 2^-60 and K + K roundings of 2^-53 (as in
the other tests of the form)."""
import math
from fractions import Fraction

import numpy as np
import pytest
import torch

import lentil_gb300 as lg

pytestmark = pytest.mark.gpu

OUT = 256                        # outputs a side: three tiles of 96
COUNT = 16                       # fields at once: 288 tiles and more, so that a CTA sums whole runs
LARGEST = sum(255 * 2.0 ** (-9 * i) for i in range(6)) / 256
PI = np.longdouble('3.14159265358979323846264338327950288')


def _column(K):
    rng = np.random.default_rng(K)
    return sum(rng.integers(250, 256, K) * 2.0 ** (-9 * i) for i in range(6)) / 256 * 2.0 ** -3


def _sums(K, alpha, shift, offset, x):
    """sum over r of x[r] exp(-2 pi i alpha (r + offset)(u - shift)), for the outputs u."""
    re, im = [], []
    for u in range(OUT):
        y = Fraction(u - OUT // 2) - Fraction(shift)
        ph = [Fraction(alpha) * (r - K // 2 + Fraction(offset)) * y for r in range(K)]
        t = np.array([int((p - math.floor(p)) * 2 ** 64) for p in ph], dtype=object)
        a = 2 * PI * (t.astype(np.longdouble) / np.longdouble(2.0 ** 64))
        re.append((x * np.cos(a)).sum())
        im.append((-x * np.sin(a)).sum())
    return np.array(re), np.array(im)


def _transform(f, alpha, shift, offset):
    """One field's transform, done COUNT times in one call (the same bits each time)."""
    F = lg.fourier.dft2_batch(f.expand(COUNT, -1, -1).contiguous(), alpha, shape=(OUT, OUT), shift=shift, offset=offset,
                              unitary=False)
    assert all(torch.equal(F[k], F[0]) for k in range(COUNT))
    return F[0].cpu().numpy()


# one, two and four chains of 64 (the runs of groups 1 and 0), one more run begun,
# remainders of a chain and of a stage
@pytest.mark.parametrize('K', [64, 100, 128, 192, 250, 256, 320, 513])
@pytest.mark.parametrize('sign', [1, -1])
def test_largest_digits(cuda_device, K, sign):
    # cos(2 pi phase) = LARGEST at the middle output, give or take 2^-28 along the sum
    offset, y0 = float(1 << 29), 256.0
    alpha = math.acos(sign * LARGEST) / (2 * math.pi) / (offset * y0)
    x = _column(K)
    (a, b), (c, d) = _sums(K, alpha, -y0, offset, x), _sums(K, alpha, -y0, offset, np.ones(K))
    f = torch.as_tensor(np.broadcast_to(x[:, None], (K, K)) + 0j, device='cuda')
    F = _transform(f, alpha, -y0, offset)
    want = (np.outer(a, c) - np.outer(b, d), np.outer(a, d) + np.outer(b, c))
    bound = K * x.sum() * (4 * K * 2.0 ** -53)
    assert float(np.abs(F.real - want[0]).max()) <= bound
    assert float(np.abs(F.imag - want[1]).max()) <= bound


def test_digits_of_both_components(cuda_device):
    # re and im alike: (re + im) / 2, the third set, has the largest digits too
    K = 256
    offset, y0 = float(1 << 29), 256.0
    alpha = 0.125 / (offset * y0)            # cos = -sin' = 0.707..: |re + im| at its largest
    x = _column(K)
    (re, im), (c, d) = _sums(K, alpha, -y0, offset, x), _sums(K, alpha, -y0, offset, np.ones(K))
    f = torch.as_tensor(np.broadcast_to(x[:, None], (K, K)) * (1 - 1j), device='cuda')
    F = _transform(f, alpha, -y0, offset)
    a, b = np.outer(re, c) - np.outer(im, d), np.outer(re, d) + np.outer(im, c)
    bound = K * x.sum() * (8 * K * 2.0 ** -53)
    assert float(np.abs(F.real - (a + b)).max()) <= bound
    assert float(np.abs(F.imag - (b - a)).max()) <= bound
