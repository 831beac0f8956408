"""complex128 transforms of fields with infinities, which the tensor-core form
hands to a plain FP64 evaluation: the results (several vectors with infinities,
in both product orders; a PSF plan, whose matrices differ by wavelength), and
their cost, which stays below that of the plain transform."""
import numpy as np
import pytest
import torch

import lentil_gb300 as lg
from lentil_gb300 import _lib
from lentil_gb300.broadband import make_plan, plan_geometry

pytestmark = pytest.mark.gpu

INF = float('inf')


def _plain(f, M, N, alpha, shift=(0.0, 0.0), offset=(0.0, 0.0), unitary=1):
    m, n = f.shape
    F = torch.empty((M, N), dtype=torch.complex128, device='cuda')
    _lib.call('lgb_dft2_noalloc', f.data_ptr(), m, n, F.data_ptr(), M, N, *alpha, *shift, *offset, unitary,
              torch.cuda.current_stream().cuda_stream)
    return F


def _same(a, b):
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a[~a.isnan()], b[~b.isnan()])


def _field(m, n):
    g = torch.Generator(device='cuda').manual_seed(m)
    return torch.view_as_complex(torch.randn(m, n, 2, generator=g, dtype=torch.float64, device='cuda'))


# rows and columns beyond a block's 256, not a multiple of the lines at once
@pytest.mark.parametrize('shape', [(130, 300, 270, 301), (300, 130, 301, 270), (301, 66, 65, 530)])
@pytest.mark.parametrize('spots', [[(0, 0)], [(5, 6), (5, 64), (60, 6)], [(k, k) for k in range(66)]])
def test_infinities(cuda_device, shape, spots):
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    f = _field(m, n)
    for k, at in enumerate(spots):
        f[at] = (INF, complex(1.0, -INF), -INF, complex(INF, INF))[k % 4]
    F = lg.fourier.dft2(f, alpha, shape=(M, N), shift=(0.25, -0.5), offset=(2, -3))
    ref = _plain(f, M, N, alpha, (0.25, -0.5), (2.0, -3.0))
    assert _same(torch.view_as_real(F), torch.view_as_real(ref))


def test_cost(cuda_device):
    n = 512
    f = _field(n, n)
    f[100, 200] = INF
    alpha = (0.7 / n, 0.6 / n)

    def ms(fn):
        best = INF
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    assert ms(lambda: lg.fourier.dft2(f, alpha, shape=(n, n))) <= ms(lambda: _plain(f, n, n, alpha))


def test_infinite_amplitude_in_a_plan(cuda_device):
    npix, waves = 160, np.array([5e-7, 6e-7, 7e-7])
    box = (slice(3, 153), slice(5, 155))
    geo = plan_geometry((npix, npix), box, [], (1 / npix, 1 / npix), 10.0, lg.pupil, waves, 5e-6, shape=64, oversample=2)
    plan = make_plan(geo, precision='fp64')
    g = torch.Generator(device='cuda').manual_seed(2)
    amp = torch.rand(1, npix, npix, generator=g, dtype=torch.float64, device='cuda')
    opd = 1e-7 * torch.rand(1, npix, npix, generator=g, dtype=torch.float64, device='cuda')
    amp[0, 80, 90], amp[0, 81, 20] = INF, -INF
    w = torch.tensor([[0.2, 0.3, 0.5]], dtype=torch.float64, device='cuda')
    image = plan.execute(amp, opd, w)[0]
    ref = torch.zeros_like(image)
    M, N = geo.window_shape
    r, c = geo.window_origin
    for k, lam in enumerate(waves):
        x = 2 * np.pi * opd[0][box] / lam
        a = amp[0][box]
        F = _plain(torch.complex(a * x.cos(), a * x.sin()).contiguous(), M, N, geo.alphas[k], geo.shifts[k],
                   tuple(float(v) for v in geo.offset))
        ref[r:r + M, c:c + N] += float(w[0, k]) * (F.real ** 2 + F.imag ** 2)
    assert not bool(ref[r:r + M, c:c + N].isfinite().any())
    assert _same(image, ref)
