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

from lentil_gb300 import _lib

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
