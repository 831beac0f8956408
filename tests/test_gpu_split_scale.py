"""The power-of-two scale of the split-fp16 operands, from the largest component
of each field of a batch, wherever it lies: a field times a power of two gives
the transform times it, bit for bit, and a component 2^20 above the others does
not overflow fp16 (65504)."""
import pytest
import torch

import lentil_gb300 as lg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(8, 9), (128, 256), (181, 182), (257, 300)])   # blocks without entries; even
@pytest.mark.parametrize('count', [1, 4, 5])                                      # and odd rounds of 256 threads
def test_scale_of_each_field(cuda_device, shape, count):
    m, n = shape
    g = torch.Generator(device='cuda').manual_seed(m + count)
    r = lambda: torch.rand(count, m, n, generator=g, dtype=torch.float64, device='cuda')
    f = torch.complex(r(), r())
    for k, (i, j) in enumerate([(0, 0), (m - 1, n - 1), (m // 2, 0), (0, n - 1), (m - 1, 0)][:count]):
        f[k, i, j] = -2.0 ** 20 if k % 2 else 1j * 2.0 ** 20
    by = torch.tensor([2.0 ** e for e in (-40, 31, 0, 60, -61)][:count], dtype=torch.float64, device='cuda')
    run = lambda x: lg.fourier.dft2_batch(x, (0.01, 0.012), shape=(48, 56), shift=(0.25, -0.5),
                                          precision='split-fp16')
    a, b = run(f), run(f * by[:, None, None])
    assert bool(torch.view_as_real(a).isfinite().all())
    assert torch.equal(b, a * by[:, None, None])


def test_zero_and_non_finite_fields(cuda_device):
    f = torch.ones(3, 40, 50, dtype=torch.complex128, device='cuda')
    f[1] = 0
    f[2, 3, 4] = float('nan')
    F = lg.fourier.dft2_batch(f, 0.01, shape=(32, 32), precision='split-fp16')
    assert bool(torch.view_as_real(F[0]).isfinite().all()) and float(F[1].abs().max()) == 0.0
    assert bool(torch.view_as_real(F[2]).isnan().any())
