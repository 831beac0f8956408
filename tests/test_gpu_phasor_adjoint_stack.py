"""The stacked phasor adjoint writes the planes that the single one adds to
zeros, for planes and stacks beyond the 65535 blocks of a grid dimension too."""
import pytest
import torch

from lentil_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('count,H,W,m,n,r0,c0', [(3, 17, 140, 9, 131, 5, 2), (2, 65540, 3, 9, 2, 65531, 1),
                                                 (65537, 3, 2, 2, 2, 1, 0)])
def test_stack_equals_its_planes(cuda_device, count, H, W, m, n, r0, c0):
    g = torch.Generator(device='cuda').manual_seed(H)
    c128 = lambda: torch.view_as_complex(torch.randn(count, m, n, 2, generator=g, dtype=torch.float64, device='cuda'))
    q, f = c128(), c128()
    s = torch.cuda.current_stream().cuda_stream
    out = torch.full((count, H, W), 7.0, dtype=torch.float64, device='cuda')
    _lib.call('lgb_phasor_adjoint_stack', q.data_ptr(), f.data_ptr(), count, m, n, 6e-7, out.data_ptr(), H, W, r0, c0, s)
    for k in (0, 1, count // 2, count - 1):
        one = torch.zeros(H, W, dtype=torch.float64, device='cuda')
        _lib.call('lgb_phasor_adjoint', q[k].data_ptr(), f[k].data_ptr(), m, n, 6e-7, one.data_ptr(), W, r0, c0, s)
        assert torch.equal(out[k], one)
