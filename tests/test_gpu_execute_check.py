"""``PSFPlan.execute(check=True)``, the default, returns when the image is there,
so that an error of the device is raised by the call it belongs to; with
``check=False`` it does not wait."""
import numpy as np
import pytest
import torch

import lentil_gb300 as lg
from lentil_gb300.broadband import make_plan, plan_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['split-bf16', 'fp64'])
@pytest.mark.parametrize('npix', [64, 192])           # plain FP64 and tensor-core products
def test_check_waits(cuda_device, precision, npix):
    box = (slice(0, npix), slice(0, npix))
    geo = plan_geometry((npix, npix), box, [], (1 / npix, 1 / npix), 10.0, lg.pupil, np.array([6e-7, 7e-7]), 5e-6,
                        shape=npix // 2, oversample=2)
    plan = make_plan(geo, precision=precision)
    amp = torch.ones(1, npix, npix, dtype=torch.float64, device='cuda')
    opd, w = torch.zeros_like(amp), torch.ones(1, 2, dtype=torch.float64, device='cuda')
    plan.execute(amp, opd, w)                          # (kernels loaded)
    stream = torch.cuda.current_stream()
    torch.cuda._sleep(100_000_000)                     # some 50 ms
    plan.execute(amp, opd, w, check=False)
    assert not stream.query()
    plan.execute(amp, opd, w)
    assert stream.query()
