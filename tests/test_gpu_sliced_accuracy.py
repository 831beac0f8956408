"""The complex128 tensor-core form leaves a transform no further from exact than
the plain FP64 GEMMs (``lgb_dft2_noalloc``), on fields of one size of amplitude
and on those that fixed-point digits suit least: a cross of ones over 1e-3, a line
of ones over 1e-4 across the longer side, and amplitudes over ten decades.

Exact: the same transform in extended precision (``np.longdouble``, at least 64
bits of mantissa) over some of its rows.  Errors are root-mean-square over those
rows, of some 1e4 roundings: 1.1 leaves room for their scatter."""
import numpy as np
import pytest
import torch

import lentil_gb300 as lg
from lentil_gb300 import _lib

pytestmark = pytest.mark.gpu

PI = np.longdouble('3.14159265358979323846264338327950288')


def _field(kind, m, n):
    rng = np.random.default_rng(m + n)
    r = lambda: rng.standard_normal((m, n))
    if kind == 'random':
        return r() + 1j * r()
    if kind == 'cross':
        f = 1e-3 * (r() + 1j * r())
        f[m // 2, :] += 1
        f[:, n // 2] += 1
        return f
    if kind == 'line':
        f = 1e-4 * (r() + 1j * r())
        f[(slice(None), n // 3) if m <= n else (m // 3, slice(None))] += 1
        return f
    return r() * np.exp(6 * r()) + 1j * (r() * np.exp(6 * r()))


def _matrix(rows, length, count, alpha):
    """exp(-2 pi i alpha u r) for the given output rows u, as (cos, -sin)."""
    y = (np.asarray(rows) - count // 2).astype(np.longdouble)[:, None]
    x = (np.arange(length) - length // 2).astype(np.longdouble)[None]
    ph = np.longdouble(alpha) * (y * x)
    ph = 2 * PI * (ph - np.rint(ph))
    return np.cos(ph), -np.sin(ph)


def _product(a, b):
    return a[0] @ b[0] - a[1] @ b[1], a[0] @ b[1] + a[1] @ b[0]


@pytest.mark.parametrize('kind', ['random', 'cross', 'decades', 'line'])
@pytest.mark.parametrize('shape', [(128, 128, 128, 128), (256, 256, 256, 256), (333, 257, 290, 301),
                                   (8, 1040, 8, 260), (1040, 8, 260, 8), (32, 800, 400, 49)])     # long sums
def test_no_further_from_exact_than_fp64(cuda_device, shape, kind):
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    f = _field(kind, m, n)
    rows = np.arange(0, M, max(1, M // 48))
    ld = lambda z: (z.real.astype(np.longdouble), z.imag.astype(np.longdouble))
    t = _product(_matrix(rows, m, M, alpha[0]), ld(f))
    e2 = _matrix(np.arange(N), n, N, alpha[1])
    ref = _product(t, (e2[0].T, e2[1].T))

    fd = torch.as_tensor(f, device='cuda')
    sliced = lg.fourier.dft2(fd, alpha, shape=(M, N), unitary=False)
    plain = torch.empty_like(sliced)
    _lib.call('lgb_dft2_noalloc', fd.data_ptr(), m, n, plain.data_ptr(), M, N, *alpha, 0.0, 0.0, 0.0, 0.0, 0,
              torch.cuda.current_stream().cuda_stream)

    def error(F):
        z = F.cpu().numpy()[rows]
        return float(np.sqrt(np.mean((z.real - ref[0]) ** 2 + (z.imag - ref[1]) ** 2)))
    assert error(sliced) <= 1.1 * error(plain), (error(sliced), error(plain))
