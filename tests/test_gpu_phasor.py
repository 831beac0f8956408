"""The phasor kernels' cosines and sines against long double, component by
component: at the axes, next to them at any distance, between the points of
the table, beyond 2^11 and 2^52 half-cycles, and for zero, infinite and NaN
phases."""
import numpy as np
import pytest
import torch

from lentil_gb300 import _device as dv
from lentil_gb300 import _lib

pytestmark = pytest.mark.gpu

PI = np.longdouble('3.14159265358979323846264338327950288')


def _reference(x):
    """(cos, sin)(pi x), reduced exactly to |t| <= 1/4 first."""
    x = np.fmod(x, 2.0)
    q = np.rint(2 * x)
    t = PI * (x.astype(np.longdouble) - q / 2)
    c, s = np.cos(t), np.sin(t)
    k = q.astype(int) % 4
    return (np.choose(k, [c, -s, -c, s]), np.choose(k, [s, c, -s, -c]))


def _phases(kind):
    rng = np.random.default_rng(17)
    if kind == 'axes':
        return np.concatenate([np.arange(-9, 9) / 2, [2.0 ** 52 + 1, 2.0 ** 53 + 2, 2.0 ** 80, -2.0 ** 60]])
    sign = rng.choice([-1.0, 1.0], 4000)
    if kind == 'near':
        return rng.integers(-6, 7, 4000) / 2 + sign * 10 ** rng.uniform(-16, -1, 4000)
    if kind == 'tiny':
        return sign * 10 ** rng.uniform(-300, 0, 4000)
    if kind == 'table':                                  # the table's points and half-way between
        return np.arange(-1024, 1025) / 512.0 + rng.choice([-1e-13, 0.0, 1e-13], 2049)
    return sign * 10 ** rng.uniform(0, 15, 4000)


@pytest.mark.parametrize('kind', ['axes', 'near', 'tiny', 'table', 'large'])
def test_phasor_components(cuda_device, kind):
    x = _phases(kind)
    opd = torch.as_tensor(x, device='cuda')
    out = torch.empty(len(x), dtype=torch.complex128, device='cuda')
    _lib.call('lgb_phasor', None, 1.0, None, opd.data_ptr(), 0.0, 1, len(x), 0, 0, 1, len(x), 2.0,
              out.data_ptr(), dv.stream_ptr())             # amplitude 1, 2 / wavelength 1
    got = out.cpu().numpy()
    for g, r in zip((got.real, got.imag), _reference(x)):
        # 2^-60 of the fixed-point value over its smallest, 2^-7.35, and the
        # rounding to double
        assert np.all(np.abs(g - r) <= 2.6e-16 * np.abs(r))


def test_phasor_non_finite(cuda_device):
    x = torch.tensor([float('inf'), float('-inf'), float('nan'), 0.25], dtype=torch.float64, device='cuda')
    out = torch.empty(4, dtype=torch.complex128, device='cuda')
    _lib.call('lgb_phasor', None, 1.0, None, x.data_ptr(), 0.0, 1, 4, 0, 0, 1, 4, 2.0, out.data_ptr(),
              dv.stream_ptr())
    got = out.cpu().numpy()
    assert np.all(np.isnan(got[:3].real) & np.isnan(got[:3].imag)) and np.isfinite(got[3])


@pytest.mark.parametrize('amp', [1.0, -0.7310585786300049, 3e300, 2e-290, 5e-324, 0.0, float('inf'), float('nan')])
def test_phasor_amplitude(cuda_device, amp):
    x = np.concatenate([_phases('axes'), _phases('near')[:500], _phases('table')[:500]])
    opd = torch.as_tensor(x, device='cuda')
    a = torch.full((len(x),), amp, dtype=torch.float64, device='cuda')
    out = torch.empty(len(x), dtype=torch.complex128, device='cuda')
    _lib.call('lgb_phasor', a.data_ptr(), 0.0, None, opd.data_ptr(), 0.0, 1, len(x), 0, 0, 1, len(x), 2.0,
              out.data_ptr(), dv.stream_ptr())
    got = out.cpu().numpy()
    with np.errstate(all='ignore'):
        for g, r in zip((got.real, got.imag), _reference(x)):
            want = np.longdouble(amp) * r
            ok = np.isfinite(want)
            assert np.array_equal(np.isnan(g), np.isnan(want)) and np.array_equal(np.isinf(g), np.isinf(want))
            # as above; subnormal results have an absolute last place
            assert np.all(np.abs(g[ok] - want[ok]) <= 2.6e-16 * np.abs(want[ok]) + 5e-324)
