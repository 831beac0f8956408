"""complex128 dft2 on the tensor cores (digit slicing): tile and K remainders,
both product orders, batches, extreme scales, and non-finite input, against
the plain FP64 evaluation of the same transform (``lgb_dft2_noalloc`` never
takes the sliced form).

Bound: K rounding errors of 2^-53 at most on either side of a sum of K terms,
K the longer contraction, relative to the output's peak."""
import numpy as np
import pytest
import torch

import lentil_gb300 as lg
from lentil_gb300 import _lib

pytestmark = pytest.mark.gpu

# (m, n, M, N): 48-column and 128-row tiles, 32-entry K stages, and their
# neighbours; the smallest shapes of the rule; wide and tall transforms (the
# right and the left product order); all of them take the sliced form
SHAPES = [(96, 96, 96, 96), (97, 129, 95, 96), (127, 128, 129, 144), (160, 95, 47, 260),
          (33, 257, 190, 193), (300, 64, 97, 128), (64, 300, 128, 97), (32, 800, 400, 49), (8, 1040, 8, 260), (8, 9, 600, 600),
          (255, 256, 257, 241)]


def _plain(f, M, N, alpha, shift, offset, unitary=1):
    m, n = f.shape
    F = torch.empty((M, N), dtype=torch.complex128, device='cuda')
    _lib.check(_lib.load().lgb_dft2_noalloc(f.data_ptr(), m, n, F.data_ptr(), M, N, *alpha, *shift,
                                            *offset, unitary,
                                            torch.cuda.current_stream().cuda_stream))
    return F


def _field(m, n, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    r = lambda: torch.randn(m, n, generator=g, dtype=torch.float64, device='cuda')
    return torch.complex(r(), r())


ARGS = dict(shift=(1.375, -0.25), offset=(2, -3))


@pytest.mark.parametrize('shape', SHAPES)
def test_matches_plain_fp64(cuda_device, shape):
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    bound = max(m, n) * 2 * 2.0 ** -53
    f = _field(m, n, m + n)
    ref = _plain(f, M, N, alpha, ARGS['shift'], ARGS['offset'])
    for k in range(2):                        # without and with a cached plan
        F = lg.fourier.dft2(f, alpha, shape=(M, N), **ARGS)
        assert float((F - ref).abs().max()) <= bound * float(ref.abs().max())
    # a batch gives each field's transform, whatever the others are
    fs = torch.stack([f, 1e-200 * f.conj(), torch.zeros_like(f), 1e200 * f])
    Fs = lg.fourier.dft2_batch(fs, alpha, shape=(M, N), **ARGS)
    for k in range(4):
        one = lg.fourier.dft2(fs[k], alpha, shape=(M, N), **ARGS)
        assert torch.equal(Fs[k], one)
    assert torch.equal(Fs[0], F) and float(Fs[2].abs().max()) == 0.0
    assert float((Fs[3] / 1e200 - ref).abs().max()) <= 2 * bound * float(ref.abs().max())


def test_largest_digits(cuda_device):
    # every digit product of group 0 at its largest: alpha tiny makes E1 and E2
    # all ones, and the field is a power of two, so each sum is exact
    m = n = M = N = 288
    f = torch.full((m, n), 2.0 ** -7, dtype=torch.complex128, device='cuda')
    F = lg.fourier.dft2(f, 0.0, shape=(M, N), unitary=False)
    assert bool((F == m * n * 2.0 ** -7).all())
    f = f * (1 - 2.0 ** -53)                  # all digits of the field in use
    F = lg.fourier.dft2(f, 0.0, shape=(M, N), unitary=False)
    exact = m * n * 2.0 ** -7 * (1 - 2.0 ** -53)
    assert float((F.real - exact).abs().max()) <= 2 * 2.0 ** -53 * exact


@pytest.mark.parametrize('bad', [float('nan'), float('inf'), -float('inf'), complex(float('inf'), float('inf'))])
@pytest.mark.parametrize('shape', [(100, 131, 120, 97), (160, 100, 90, 260)])
def test_non_finite_input(cuda_device, bad, shape):
    # the same infinities and NaNs as the plain evaluation, in the one field
    # that holds them
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    f = _field(m, n, 3)
    f[m // 3, n // 2] = bad
    good = _field(m, n, 4)
    ref = _plain(f, M, N, alpha, ARGS['shift'], ARGS['offset'])
    F = lg.fourier.dft2_batch(torch.stack([good, f, good]), alpha, shape=(M, N), **ARGS)
    a, b = torch.view_as_real(F[1]), torch.view_as_real(ref)
    assert torch.equal(a.isnan(), b.isnan())
    assert torch.equal(a[~a.isnan()], b[~b.isnan()])          # signed infinities
    assert torch.equal(F[0], F[2]) and bool(torch.view_as_real(F[0]).isfinite().all())


@pytest.mark.parametrize('shape', [(1, 1, 1, 1), (5, 3, 2, 7), (15, 17, 16, 33), (64, 8, 9, 130),
                                   (7, 300, 300, 7), (100, 90, 80, 70)])
def test_plain_small_shapes(cuda_device, shape):
    # the plain form's 16 x 16 tiles and 8-entry K blocks, split and whole,
    # against the oracle; a batch splits K differently, to rounding
    from oracle import lentil_oracle as lo
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    f = _field(m, n, 8)
    ref = lo.dft2(f.cpu().numpy(), alpha, shape=(M, N), **ARGS)
    for k in range(2):
        F = lg.fourier.dft2(f, alpha, shape=(M, N), **ARGS)
        assert lo.peak_normalised_error(F.cpu().numpy(), ref) < 1e-13
    Fs = lg.fourier.dft2_batch(torch.stack([f] * 40), alpha, shape=(M, N), **ARGS)
    assert float((Fs - F).abs().max()) <= 1e-14 * float(F.abs().max())


def test_rule_is_by_shape(cuda_device):
    # the form depends on the shape alone, so a workspace query, a plan and a
    # one-off transform agree on it on every machine
    lib = _lib.load()
    small, large = (64, 64, 128, 128), (128, 128, 128, 128)
    plain = 16 * (128 * 64 + 64 * 128 + max(128 * 64, 64 * 128))
    assert lib.lgb_dft2_workspace_size(*small, _lib.FP64) - plain < 1024
    assert lib.lgb_dft2_workspace_size(*large, _lib.FP64) > 4 * 128 * 128 * 16


@pytest.mark.parametrize('n,os_', [(65, 1), (96, 5), (97, 2), (127, 3), (130, 70), (193, 2), (257, 4)])
def test_pixelate_products(cuda_device, n, os_):
    # sizes around the 96-row windows of the banded products and the 64-entry
    # chains, with zeroed rows (the mask) and one bright pixel
    from oracle import lentil_oracle as lo
    rng = np.random.default_rng(n)
    img = rng.random((n, n))
    img[:3], img[:, -2:], img[n // 2, n // 3] = 0, 0, 1e3
    assert lo.peak_normalised_error(lg.detector.pixel(img, os_), lo.pixel(img, os_)) < 1e-13
    ref = lo.pixelate(img, os_)
    # the rescaling divides by the sum of the samples, which a large
    # oversampling of few samples makes small: scale the bound by it
    assert lo.peak_normalised_error(lg.detector.pixelate(img, os_), ref) < 1e-12


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
def test_pixelate_of_non_finite_images(cuda_device, bad):
    rng = np.random.default_rng(2)
    img = rng.random((100, 100))
    img[3, 4] = bad
    for os_ in (2, 3):
        assert np.isnan(lg.detector.pixelate(img, os_)).all()
    p = lg.detector.pixel(img, 2)
    assert not np.isfinite(p).any()
    assert np.isfinite(lg.detector.pixelate(np.nan_to_num(img, posinf=1.0), 3)).all()


@pytest.mark.parametrize('shape', [(120, 130, 602, 601), (120, 130, 301, 257), (120, 130, 97, 130)])
def test_finish_rows(cuda_device, shape):
    # results in groups of four rows (the last group partly filled) and row by row
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    f = _field(m, n, 9)
    ref = _plain(f, M, N, alpha, ARGS['shift'], ARGS['offset'])
    F = lg.fourier.dft2(f, alpha, shape=(M, N), **ARGS)
    assert float((F - ref).abs().max()) <= 2 * max(m, n) * 2.0 ** -53 * float(ref.abs().max())
