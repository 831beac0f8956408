"""complex128 PSF plans whose digit matrices pass the 16 GiB that a plan keeps:
195 wavelengths of 1024 x 1024 to 1024 x 1024 stay below, 196 pass it and have
their matrices built chunk by chunk.  With no weight on the last one, the images
are the same bits (the sums behind them are integers, whatever the chunks)."""
import ctypes

import numpy as np
import pytest
import torch

from lentil_gb300 import _lib
from lentil_gb300.broadband import PSFPlan

pytestmark = pytest.mark.gpu


def _plan(waves, n=1024, batch=1):
    lam = np.linspace(5e-7, 9e-7, 196)[:waves]
    alphas = [(0.4 * 5e-7 / l / n, 0.45 * 5e-7 / l / n) for l in lam]
    return PSFPlan((n, n), (0, 0, n, n), (0, 0), lam, alphas, [(0.25, -0.5)] * waves, (n, n), (n, n), (0, 0),
                   batch=batch, precision='fp64')


def test_matrices_by_chunk(cuda_device):
    g = torch.Generator(device='cuda').manual_seed(3)
    amp = torch.rand(2, 1024, 1024, generator=g, dtype=torch.float64, device='cuda')
    opd = 1e-7 * torch.rand(2, 1024, 1024, generator=g, dtype=torch.float64, device='cuda')
    w = torch.rand(2, 196, generator=g, dtype=torch.float64, device='cuda')
    w[:, 195] = 0
    small = _plan(195, batch=2)
    assert _lib.load().lgb_psf_plan_bytes(small._h) > 17 << 30
    want = small.execute(amp, opd, w[:, :195].contiguous())
    del small
    large = _plan(196, batch=2)
    assert _lib.load().lgb_psf_plan_size(ctypes.byref(large.desc)) < 17 << 30     # fields, results, one chunk
    for _ in range(2):
        assert torch.equal(large.execute(amp, opd, w), want)
    torch.cuda.empty_cache()
