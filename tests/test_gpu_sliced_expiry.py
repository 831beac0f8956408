"""The bounded waits of the complex128 tensor-core products, run out on the GPU.

A one-shot hook makes the first CTA of one GEMM hold back a stage's loads, or
the release of a stage's leading digits, so that the producer is left with half
a stage in flight.  Every wait is bounded by 1 ms then: the launch must retire
what it issued and return, the transform must come out as the plain FP64 form
gives it (``lgb_dft2_noalloc``), and the next call must be normal again, bit for
bit.

Bound: as in the tests of the sliced form, K rounding errors of 2^-53 on either
side."""
import time

import pytest
import torch

import lentil_gb300 as lg
from lentil_gb300 import _lib
from lentil_gb300.broadband import PSFPlan

pytestmark = pytest.mark.gpu

ARGS = (1.375, -0.25, 2.0, -3.0, 1)


def _run(entry, f, M, N, alpha, *more):
    m, n = f.shape
    F = torch.empty((M, N), dtype=torch.complex128, device='cuda')
    _lib.call(entry, f.data_ptr(), m, n, F.data_ptr(), M, N, *alpha, *ARGS, *more,
              torch.cuda.current_stream().cuda_stream)
    return F


# the stages of a CTA run on from tile to tile; a release withheld at stage s
# stops the loads of stage s + 2 halfway
@pytest.mark.parametrize('launch', [0, 1])
@pytest.mark.parametrize('release,stage', [(0, 0), (0, 5), (1, 0), (1, 5)])
@pytest.mark.parametrize('shape', [(512, 520, 500, 530), (520, 512, 530, 500)])     # (E1 f) E2, E1 (f E2)
def test_withheld_stage(cuda_device, shape, release, stage, launch):
    lib = _lib.load()
    m, n, M, N = shape
    alpha = (0.7 / max(m, M), 0.6 / max(n, N))
    g = torch.Generator(device='cuda').manual_seed(m)
    f = torch.view_as_complex(torch.randn(m, n, 2, generator=g, dtype=torch.float64, device='cuda'))
    nbytes = lib.lgb_dft2_workspace_size(m, n, M, N, _lib.FP64)
    ws = torch.empty(nbytes, dtype=torch.uint8, device='cuda')
    sliced = lambda: _run('lgb_dft2', f, M, N, alpha, _lib.FP64, ws.data_ptr(), nbytes)
    plain = _run('lgb_dft2_noalloc', f, M, N, alpha)
    before = sliced()
    torch.cuda.synchronize()

    _lib.check(lib.lgb_test_stall_sliced(launch, stage, release, 1.0))
    t0 = time.perf_counter()
    F = sliced()
    torch.cuda.synchronize()
    elapsed = time.perf_counter() - t0
    assert elapsed < 1.0, elapsed                      # about 1 ms, not the 2 s default
    word = ws[:4].view(torch.int32)
    assert int(word) == _lib.ETIMEOUT                  # the wait did run out
    bound = 2 * max(m, n) * 2.0 ** -53 * float(plain.abs().max())
    assert float((F - plain).abs().max()) <= bound

    again = sliced()
    assert int(word) == _lib.OK
    assert torch.equal(again, before)


def _stalled(call, launch, release, stage):
    _lib.check(_lib.load().lgb_test_stall_sliced(launch, stage, release, 1.0))
    t0 = time.perf_counter()
    out = call()
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 1.0
    return out


@pytest.mark.parametrize('launch', [0, 1])
@pytest.mark.parametrize('release,stage', [(0, 3), (1, 3)])
def test_plan_with_matrices_by_wavelength(cuda_device, release, stage, launch):
    n, waves = 384, 5
    lam = [5e-7 + 5e-8 * k for k in range(waves)]
    plan = PSFPlan((n, n), (0, 0, n, n), (0, 0), lam, [(0.5 * 5e-7 / l / n, 0.4 * 5e-7 / l / n) for l in lam],
                   [(0.25, -0.5)] * waves, (n, n), (n, n), (0, 0), precision='fp64')
    g = torch.Generator(device='cuda').manual_seed(9)
    amp = torch.rand(1, n, n, generator=g, dtype=torch.float64, device='cuda')
    opd = 1e-7 * torch.rand(1, n, n, generator=g, dtype=torch.float64, device='cuda')
    w = torch.rand(1, waves, generator=g, dtype=torch.float64, device='cuda')
    run = lambda: plan.execute(amp, opd, w, check=False)
    before = run()
    image = _stalled(run, launch, release, stage)
    assert not torch.equal(image, before)              # in plain FP64: other roundings
    # an |F| of at most amp.sum() is off by 4 n roundings of it
    assert float((image - before).abs().max()) <= waves * 2 * 4 * n * 2.0 ** -53 * float(before.max())
    assert torch.equal(run(), before)


@pytest.mark.parametrize('launch', [0, 1])
@pytest.mark.parametrize('release,stage', [(0, 2), (1, 2)])
def test_pixel_products(cuda_device, release, stage, launch):
    n = 700
    g = torch.Generator(device='cuda').manual_seed(9)
    img = torch.rand(n, n, generator=g, dtype=torch.float64, device='cuda')
    run = lambda: lg.detector.pixel(img, 3)
    before = run()
    image = _stalled(run, launch, release, stage)
    assert not torch.equal(image, before)
    assert float((image - before).abs().max()) <= 4 * n * 2.0 ** -53 * float(before.max())
    assert torch.equal(run(), before)
