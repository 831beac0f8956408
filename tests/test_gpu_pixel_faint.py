"""The pixel MTF keeps pixels that are faint beside their row as accurate as FP64
products with the same circulant matrices do: relative to themselves, not to the
brightest pixel.

The images are a core of 1 over a background; reference: extended precision
(``np.longdouble``) from taps of that precision; comparison: the two products by
numpy in double precision, from taps in double precision.  The median over the
pixels counts: half of them lie in rows and columns that miss the core.  Both
medians come from errors of a few units of 2^-53 in taps and sums: a factor of
two between them is scatter, losing the background's digits a factor of 1e3."""
import numpy as np
import pytest

import lentil_gb300 as lg

pytestmark = pytest.mark.gpu

PI = np.longdouble('3.14159265358979323846264338327950288')


def _taps(N, os_, T):
    """ifft(sinc(fftfreq(N) os)) in the type T, the phases reduced in integers."""
    f = np.fft.fftshift(np.arange(N) - N // 2)
    num = f * os_
    with np.errstate(invalid='ignore'):
        s = np.where(num == 0, T(1), np.sin(T(PI) * ((num % (2 * N)).astype(T) / N)) / (T(PI) * (num.astype(T) / N)))
    phase = (np.outer(np.arange(N), f) % N).astype(T)
    return (np.cos(2 * T(PI) * phase / N) * s).sum(axis=1) / N


@pytest.mark.parametrize('background', [1e-7, 1e-10])
@pytest.mark.parametrize('N,os_', [(150, 2), (150, 3), (321, 3)])
def test_faint_pixels(cuda_device, N, os_, background):
    y = np.arange(N) - N // 2
    img = np.exp(-(y[:, None] ** 2 + y[None, :] ** 2) / 8.0) + background
    at = (y[:, None] - y[None, :]) % N
    C = _taps(N, os_, np.longdouble)[at]
    ref = np.abs(C @ img.astype(np.longdouble) @ C.T)
    D = _taps(N, os_, np.float64)[at]
    error = lambda p: float(np.median(np.abs(p - ref) / ref))
    assert error(lg.detector.pixel(img, os_)) <= 2 * error(np.abs(D @ img @ D.T))


@pytest.mark.parametrize('N', [65, 127, 150])          # odd tiles of 32; windows that wrap at both ends
def test_one_pixel_spreads_by_the_taps(cuda_device, N):
    # |c(k) c(l)| around the pixel, wherever it lies: every pixel to its own last places
    c = np.abs(_taps(N, 3, np.longdouble))
    for at in ((0, 0), (N - 1, N // 2), (N // 3, N - 2)):
        img = np.zeros((N, N))
        img[at] = 3.0
        k, l = (np.arange(N) - at[0]) % N, (np.arange(N) - at[1]) % N
        ref = 3 * np.outer(c[k], c[l])
        # taps are sums of N terms of at most 1/N: N 2^-53 of it each at most
        bound = 3 * (c[k][:, None] + c[l][None, :] + 2.0 ** -53) * 2 * 2.0 ** -53 + 4 * 2.0 ** -53 * ref
        assert bool((np.abs(lg.detector.pixel(img, 3) - ref) <= bound).all())
