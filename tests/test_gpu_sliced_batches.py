"""Batches of the complex128 tensor-core form that are done in several chunks
(512 MB of digits and sums): each member is the transform of its own, bit for
bit, with shared matrices and with the plan's of each wavelength."""
import numpy as np
import pytest
import torch

import lentil_gb300 as lg
from lentil_gb300 import _lib
from lentil_gb300.broadband import PSFPlan

pytestmark = pytest.mark.gpu


# members of some 107, 28 and 28 MB: chunks of four and three, of 18 and 17, one over
@pytest.mark.parametrize('shape,count', [((1019, 941, 1024, 1024), 7), ((512, 512, 512, 512), 35),
                                         ((500, 530, 520, 512), 19)])
def test_shared_matrices(cuda_device, shape, count):
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    one = _lib.load().lgb_dft2_batch_workspace_size(1, *shape, _lib.FP64)
    assert _lib.load().lgb_dft2_batch_workspace_size(count, *shape, _lib.FP64) < count * one     # not all at once
    g = torch.Generator(device='cuda').manual_seed(count)
    f = torch.view_as_complex(torch.randn(count, m, n, 2, generator=g, dtype=torch.float64, device='cuda'))
    for _ in range(2):                         # without and with a cached plan
        F = lg.fourier.dft2_batch(f, alpha, shape=(M, N), shift=(0.5, -0.25))
    for k in range(count):
        assert torch.equal(F[k], lg.fourier.dft2(f[k], alpha, shape=(M, N), shift=(0.5, -0.25)))


def test_matrices_of_each_wavelength(cuda_device):
    n, waves = 1000, 7
    lam = np.linspace(5e-7, 8e-7, waves)
    alphas = [(0.5 * 5e-7 / l / n, 0.4 * 5e-7 / l / n) for l in lam]
    plan = lambda k: PSFPlan((n, n), (0, 0, n, n), (0, 0), lam[k], [alphas[i] for i in range(waves)[k]],
                             [(0.25, -0.5)] * len(lam[k]), (n, n), (n, n), (0, 0), precision='fp64')
    g = torch.Generator(device='cuda').manual_seed(1)
    amp = torch.rand(1, n, n, generator=g, dtype=torch.float64, device='cuda')
    opd = 1e-7 * torch.rand(1, n, n, generator=g, dtype=torch.float64, device='cuda')
    w = torch.rand(1, waves, generator=g, dtype=torch.float64, device='cuda')
    image = plan(slice(0, waves)).execute(amp, opd, w)
    ref = torch.zeros_like(image)
    for k in range(waves):
        plan(slice(k, k + 1)).execute(amp, opd, w[:, k:k + 1].contiguous(), out=ref, accumulate=True)
    # the same |F|^2; their weighted sum is rounded in another order
    assert float((image - ref).abs().max()) <= 2 * waves * 2.0 ** -53 * float(ref.abs().max())
