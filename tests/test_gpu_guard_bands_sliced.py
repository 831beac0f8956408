"""Write-bounds checks, as in ``test_gpu_guard_bands.py``, of the complex128
tensor-core form: results, workspace and plan memory between sentinel margins,
for shapes with remainders of every tile, both product orders, and batches in
one and several chunks.  Every shape is above the rule's 2 x 96^3 multiply-adds."""
import ctypes

import numpy as np
import pytest
import torch

from lentil_gb300 import _lib
from tests.test_gpu_guard_bands import Guarded, _c128, _s

pytestmark = pytest.mark.gpu

ARGS = (0.0021, 0.0023, 0.5, -1.0, 1.0, 2.0, 1)
SHAPES = [(97, 129, 95, 96), (129, 97, 96, 125), (33, 257, 190, 193), (257, 33, 193, 190), (8, 1040, 8, 260),
          (1040, 8, 260, 8), (8, 9, 600, 600), (255, 256, 257, 241)]


def _sliced(shape):
    m, n, M, N = shape
    plain = 16 * (M * m + n * N + max(M * n, m * N))
    return _lib.load().lgb_dft2_workspace_size(m, n, M, N, _lib.FP64) > plain + 4096


@pytest.mark.parametrize('shape', SHAPES)
@pytest.mark.parametrize('count', [1, 3])
def test_batch(cuda_device, shape, count):
    assert _sliced(shape)
    m, n, M, N = shape
    lib = _lib.load()
    f = _c128((count, m, n), m * n)
    F = Guarded(16 * count * M * N)
    nbytes = lib.lgb_dft2_batch_workspace_size(count, m, n, M, N, _lib.FP64)
    ws = Guarded(nbytes)
    _lib.call('lgb_dft2_batch', f.data_ptr(), count, m, n, F.ptr, M, N, *ARGS, _lib.FP64, ws.ptr, nbytes, _s())
    F.check()
    ws.check()
    f[0, m // 2, n // 3] = float('inf')         # the plain evaluation, in the same workspace
    _lib.call('lgb_dft2_batch', f.data_ptr(), count, m, n, F.ptr, M, N, *ARGS, _lib.FP64, ws.ptr, nbytes, _s())
    F.check()
    ws.check()


def test_batch_in_chunks(cuda_device):
    m, n, M, N, count = 500, 530, 520, 509, 20          # some 28 MB each, 512 MB a chunk
    lib = _lib.load()
    f = _c128((count, m, n), 3)
    F = Guarded(16 * count * M * N)
    nbytes = lib.lgb_dft2_batch_workspace_size(count, m, n, M, N, _lib.FP64)
    ws = Guarded(nbytes)
    _lib.call('lgb_dft2_batch', f.data_ptr(), count, m, n, F.ptr, M, N, *ARGS, _lib.FP64, ws.ptr, nbytes, _s())
    F.check()
    ws.check()


@pytest.mark.parametrize('shape', SHAPES)
def test_plan(cuda_device, shape):
    m, n, M, N = shape
    lib = _lib.load()
    size = lib.lgb_dft2_plan_size(m, n, M, N, _lib.FP64)
    mem = Guarded(size)
    h = ctypes.c_void_p()
    _lib.call('lgb_dft2_plan_create_in', m, n, M, N, *ARGS, _lib.FP64, mem.ptr, size, _s(), ctypes.byref(h))
    try:
        for count in (1, 4):
            f = _c128((count, m, n), count)
            F = Guarded(16 * count * M * N)
            nbytes = lib.lgb_dft2_plan_workspace_size(h, count)
            ws = Guarded(nbytes)
            _lib.call('lgb_dft2_plan_execute', h, f.data_ptr(), count, F.ptr, ws.ptr, nbytes, _s())
            F.check()
            ws.check()
        mem.check()
    finally:
        torch.cuda.synchronize()
        lib.lgb_dft2_plan_destroy(h)


@pytest.mark.parametrize('shape', [(97, 129, 95, 96), (255, 256, 257, 241)])
def test_idft2(cuda_device, shape):
    m, n, M, N = shape
    lib = _lib.load()
    F = _c128((m, n), 5)
    out = Guarded(16 * M * N)
    nbytes = lib.lgb_idft2_workspace_size(m, n, M, N, _lib.FP64)
    ws = Guarded(nbytes)
    _lib.call('lgb_idft2', F.data_ptr(), m, n, out.ptr, M, N, 0.003, 0.0025, 0.5, -1.0, 1, _lib.FP64, ws.ptr, nbytes,
              _s())
    out.check()
    ws.check()


@pytest.mark.parametrize('field,window,waves', [((97, 129), (95, 127), 3), ((255, 241), (257, 256), 4),
                                                ((500, 510), (520, 505), 21)])       # the last in two chunks
def test_psf_plan(cuda_device, field, window, waves):
    (m, n), (M, N) = field, window
    H, W, R, C = m + 5, n + 3, M + 7, N + 2
    lib = _lib.load()
    lam = np.linspace(5e-7, 8e-7, waves)
    alpha = 0.4 * 5e-7 / lam / max(m, n)
    zero = np.zeros(waves)
    d = _lib.PsfDesc(H=H, W=W, r0=2, c0=1, m=m, n=n, offset_r=1.0, offset_c=-2.0, M=M, N=N, out_rows=R, out_cols=C,
                     win_r0=3, win_c0=1, n_wavelengths=waves, wavelengths=lam.ctypes.data, alpha_r=alpha.ctypes.data,
                     alpha_c=alpha.ctypes.data, shift_r=zero.ctypes.data, shift_c=zero.ctypes.data, batch=2,
                     precision=_lib.FP64)
    size = lib.lgb_psf_plan_size(ctypes.byref(d))
    mem = Guarded(size)
    h = ctypes.c_void_p()
    _lib.call('lgb_psf_plan_create_in', ctypes.byref(d), mem.ptr, size, ctypes.byref(h), _s())
    try:
        rng = np.random.default_rng(m)
        amp = torch.as_tensor(rng.uniform(0, 1, (2, H, W)), device='cuda')
        opd = torch.as_tensor(rng.normal(0, 1e-7, (2, H, W)), device='cuda')
        w = torch.as_tensor(rng.uniform(0, 1, (2, waves)), device='cuda')
        for count in (2, 1):
            out = Guarded(8 * count * R * C)
            _lib.call('lgb_psf_execute_batch', h, count, amp.data_ptr(), opd.data_ptr(), w.data_ptr(), out.ptr, 0, _s())
            out.check()
        mem.check()
    finally:
        torch.cuda.synchronize()
        lib.lgb_psf_plan_destroy(h)


@pytest.mark.parametrize('n,os_', [(65, 2), (97, 3), (130, 70), (321, 4), (1000, 5), (513, 1)])
def test_pixel(cuda_device, n, os_):
    lib = _lib.load()
    img = torch.as_tensor(np.random.default_rng(n).uniform(0, 1, (n, n)), device='cuda')
    nbytes = lib.lgb_pixel_workspace_size(n, os_)
    for name, out_n in (('lgb_pixel', n), ('lgb_pixelate', lib.lgb_pixelate_size(n, os_))):
        for bad in (False, True):               # True: the plain evaluation
            if bad:
                img[1, 2] = float('nan')
            out, ws = Guarded(8 * out_n * out_n), Guarded(nbytes)
            _lib.call(name, img.data_ptr(), n, n, os_, out.ptr, ws.ptr, nbytes, _s())
            out.check()
            ws.check()
        img[1, 2] = 0.5
