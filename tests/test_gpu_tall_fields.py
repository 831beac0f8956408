"""complex128 transforms of fields with more rows than 16 x 65535, which the
product order E1 (f E2) multiplies row by row first."""
import math

import pytest
import torch

import lentil_gb300 as lg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m', [16 * 65535, 16 * 65535 + 1, 1_100_003])
def test_tall_field(cuda_device, m):
    n, M, N = 2, 3, 1
    g = torch.Generator(device='cuda').manual_seed(m)
    f = torch.view_as_complex(torch.randn(m, n, 2, generator=g, dtype=torch.float64, device='cuda'))
    alpha = (2.0 ** -21, 0.25)                # powers of two: the phases below are exact
    F = lg.fourier.dft2(f, alpha, shape=(M, N), unitary=False)
    r = torch.arange(m, dtype=torch.float64, device='cuda') - m // 2
    u = torch.arange(M, dtype=torch.float64, device='cuda') - M // 2
    ph = -2 * math.pi * torch.remainder(alpha[0] * u[:, None] * r, 1.0)
    ref = torch.polar(torch.ones_like(ph), ph) @ f @ torch.ones(n, N, dtype=torch.complex128, device='cuda')
    # one output column, at v = 0: E2 is all ones.  Both sides add m terms of unit
    # size in some order: m roundings of the partial sums, below 8 sqrt(m) here
    assert float((F - ref).abs().max()) <= m * 2.0 ** -53 * 8 * math.sqrt(m)
