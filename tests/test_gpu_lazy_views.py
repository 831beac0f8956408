"""Tensors that torch keeps as lazy views (conjugates, and imaginary parts of
conjugates, whose memory holds other values) are taken by their values."""
import pytest
import torch

import lentil_gb300 as lg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [40, 130])
@pytest.mark.parametrize('precision', ['fp64', 'split-bf16'])
def test_conjugate_field(cuda_device, n, precision):
    g = torch.Generator(device='cuda').manual_seed(n)
    f = torch.view_as_complex(torch.randn(n, n, 2, generator=g, dtype=torch.float64, device='cuda'))
    lazy = f.conj()
    assert lazy.is_conj()
    F = lambda x: lg.fourier.dft2(x, 0.7 / n, shape=(n, n), shift=(0.5, 0.0), precision=precision)
    assert torch.equal(F(lazy), F(lazy.resolve_conj())) and not torch.equal(F(lazy), F(f))


def test_negated_image(cuda_device):
    z = torch.complex(torch.zeros(64, 64, dtype=torch.float64, device='cuda'),
                      torch.rand(64, 64, dtype=torch.float64, device='cuda'))
    lazy = z.conj().imag
    assert lazy.is_neg()
    assert torch.equal(lg.detector.pixel(lazy, 2), lg.detector.pixel(lazy.resolve_neg().contiguous(), 2))
