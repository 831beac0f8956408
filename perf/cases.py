"""Performance cases of the diffraction path, through the public entry points.

Each case is one call (or one loss-and-gradient evaluation) of a user's
program: the matrix Fourier transform as lentil's ``dft2`` takes it
(complex128, the default precision), ``propagate_dft``/``propagate_fft`` of a
pupil, the gradients of an image, the phase-retrieval loss, broadband PSFs
from a plan and from one call, and detector pixelation.  ``exact`` restates
each in plain torch/numpy at 64 bits.
"""
import math

import numpy as np
import torch

import lentil_gb300 as lg
from lentil_gb300 import autodiff
from lentil_gb300.broadband import make_plan, plan_geometry

FOCAL, DU = 10.0, 5e-6            # focal length and detector pixel of the sample optics (metres)


def listed():
    return [
        # the smallest transform of a loop over little stamps: latency
        dict(name='dft2_64', kind='dft2', m=64, n=64, M=64, N=64, precision='fp64', count=1),
        # a default-precision transform of a 512-pixel disc's bounding box
        dict(name='dft2_512', kind='dft2', m=512, n=512, M=512, N=512, precision='fp64', count=1),
        # odd, rectangular, off-centre: a sub-aperture onto a detector strip
        dict(name='dft2_ragged', kind='dft2', m=749, n=523, M=611, N=877, precision='fp64',
             count=1),
        # the 1024-pixel segmented pupil's bounding box onto its 1024 x 1024 window
        dict(name='dft2_1024', kind='dft2', m=1019, n=941, M=1024, N=1024, precision='fp64',
             count=1),
        # three fields in one call on the tensor-core precision
        dict(name='dft2_split_512', kind='dft2', m=512, n=512, M=512, N=512,
             precision='split-fp16', count=3),
        # lentil's monochromatic script: numpy pupil in, numpy intensity out
        dict(name='propagate_256', kind='propagate', npix=256, det=128, wavelength=650e-9),
        # the FFT propagation of the same pupil (666 x 666), tensors resident
        dict(name='propagate_fft_256', kind='fft', npix=256, wavelength=650e-9),
        # forward and backward of one image at default precision
        dict(name='gradient_256', kind='gradient', npix=256, det=128, wavelength=633e-9),
        # focus-diverse phase retrieval: three 512-pixel images, 90 modes
        dict(name='retrieval_512', kind='retrieval', npix=512, det=256, modes=90,
             wavelength=633e-9),
        # the broadband segmented PSF from a resident plan, the largest work here
        dict(name='broadband_1024', kind='broadband', npix=1024, det=512, waves=64,
             precision='split-bf16'),
        # the broadband loop at default (complex128) accuracy in one call
        dict(name='broadband_c128_512', kind='broadband_call', npix=512, det=256, waves=8),
        # detector sampling of an oversampled image whose size is not a power of two
        dict(name='pixelate_1000', kind='pixelate', size=1000, oversample=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['dft2', 'dft2', 'dft2', 'propagate', 'fft', 'gradient', 'retrieval',
                       'broadband', 'broadband_call', 'pixelate'])
    if kind == 'dft2':
        size = _log_int(rng, 40, 1000)
        m, n, M, N = (max(8, int(size * rng.uniform(0.6, 1.02))) for _ in range(4))
        return dict(kind='dft2', m=m, n=n, M=M, N=N, count=1,
                    precision=rng.choice(['fp64', 'fp64', 'split-fp16', 'split-bf16']))
    if kind == 'propagate':
        npix = _log_int(rng, 64, 512)
        return dict(kind=kind, npix=npix, det=max(16, int(npix * rng.uniform(0.3, 0.6))),
                    wavelength=rng.randint(450, 900) * 1e-9)
    if kind == 'fft':
        return dict(kind=kind, npix=_log_int(rng, 64, 300), wavelength=rng.randint(450, 800) * 1e-9)
    if kind == 'gradient':
        npix = _log_int(rng, 64, 400)
        return dict(kind=kind, npix=npix, det=max(16, int(npix * rng.uniform(0.4, 0.6))),
                    wavelength=rng.randint(450, 900) * 1e-9)
    if kind == 'retrieval':
        npix = _log_int(rng, 128, 512)
        return dict(kind=kind, npix=npix, det=npix // 2, modes=rng.randint(10, 90),
                    wavelength=rng.randint(450, 900) * 1e-9)
    if kind == 'broadband':
        npix = _log_int(rng, 256, 1024)
        return dict(kind=kind, npix=npix, det=max(32, int(npix * rng.uniform(0.3, 0.5))),
                    waves=rng.randint(4, 64), precision=rng.choice(['split-bf16', 'split-fp16']))
    if kind == 'broadband_call':
        npix = _log_int(rng, 128, 512)
        return dict(kind=kind, npix=npix, det=max(32, int(npix * rng.uniform(0.3, 0.5))),
                    waves=rng.randint(2, 8))
    return dict(kind='pixelate', oversample=rng.randint(2, 5),
                size=rng.choice([256, 512, 1024, 2048, _log_int(rng, 200, 1200)]))


# ------------------------------------------------------------------ inputs ---
def _grid(npix):
    c = (torch.arange(npix, dtype=torch.float64, device='cuda') - npix // 2) / (npix / 2)
    return c[:, None], c[None, :]


def _disc(npix):
    """Unit-power disc that spans the array, with a linear edge of one pixel."""
    y, x = _grid(npix)
    edge = (npix / 2) * (1 - torch.sqrt(y * y + x * x)) + 0.5
    amp = edge.clamp(0, 1)
    return amp / torch.sqrt((amp * amp).sum())


def _segments(npix):
    """Unit-power aperture of 18 hexagons in two rings around an empty centre."""
    y, x = _grid(npix)
    radius = 2 * 116.8 / 1024
    apothem = radius * math.sqrt(3) / 2
    gap = 2 / npix
    pitch = 2 * apothem + 2 * gap
    amp = torch.zeros(npix, npix, dtype=torch.float64, device='cuda')
    for q in range(-2, 3):
        for r in range(-2, 3):
            if abs(q + r) > 2 or (q, r) == (0, 0):
                continue
            cy, cx = pitch * (r + q / 2), pitch * q * math.sqrt(3) / 2
            inside = torch.ones_like(amp)
            for k in range(6):
                a = math.pi / 6 + k * math.pi / 3
                d = (y - cy) * math.sin(a) + (x - cx) * math.cos(a)
                inside = torch.minimum(inside, (npix / 2 * (apothem - d) + 0.5).clamp(0, 1))
            amp = torch.maximum(amp, inside)
    return amp / torch.sqrt((amp * amp).sum())


def _modes(npix, count):
    """The first ``count`` products T_i(y) T_j(x) by order, without piston."""
    y, x = _grid(npix)
    t = [torch.ones_like(y), y]
    s = [torch.ones_like(x), x]
    while len(t) < 16:
        t.append(2 * y * t[-1] - t[-2])
        s.append(2 * x * s[-1] - s[-2])
    pairs = [(i, order - i) for order in range(1, 16) for i in range(order + 1)]
    return torch.stack([t[i] * s[j] for i, j in pairs[:count]])


def _opd(npix, seed):
    """Smooth wavefront error of tens of nanometres rms: 20 low-order modes."""
    g = torch.Generator(device='cuda').manual_seed(int(seed))
    c = 20e-9 * torch.randn(20, generator=g, dtype=torch.float64, device='cuda')
    return torch.einsum('k,khw->hw', c, _modes(npix, 20))


def _geometry(case, seed):
    """alpha, shift and offset of a ``dft2`` case: Nyquist-ish sampling and
    sub-pixel shifts (in 1/64 pixel) as a tilt gives them."""
    r = np.random.RandomState(seed % (1 << 31))
    q = r.uniform(0.3, 0.9, 2)
    alpha = (float(q[0] / max(case['m'], case['M'])), float(q[1] / max(case['n'], case['N'])))
    shift = tuple(float(v) / 64 for v in r.randint(-200, 200, 2))
    offset = tuple(int(v) for v in r.randint(-6, 7, 2))
    return alpha, shift, offset


def _fields(case, seed):
    """Pupil-like fields: a unit-power disc with smooth phase and scattered light."""
    m, n, count = case['m'], case['n'], case['count']
    g = torch.Generator(device='cuda').manual_seed(int(seed))
    y = (torch.arange(m, dtype=torch.float64, device='cuda') - m // 2)[:, None] / (m / 2)
    x = (torch.arange(n, dtype=torch.float64, device='cuda') - n // 2)[None, :] / (n / 2)
    c = 0.3 * torch.randn(count, 6, 1, 1, generator=g, dtype=torch.float64, device='cuda')
    ph = (c[:, 0] * y + c[:, 1] * x + c[:, 2] * y * x + c[:, 3] * (y * y + x * x)
          + c[:, 4] * y ** 3 + c[:, 5] * x ** 3)
    ph = ph + 0.1 * torch.randn(count, m, n, generator=g, dtype=torch.float64, device='cuda')
    amp = ((y * y + x * x) <= 1).to(torch.float64)
    f = torch.polar(amp.expand(count, m, n).contiguous(), ph)
    return f / math.sqrt(float((amp * amp).sum()))


def _weights(waves):
    lam = np.linspace(500e-9, 900e-9, waves)
    x = 0.0143877 / (lam * 5800.0)
    w = lam ** -4 / np.expm1(x)
    return lam, w / w.sum()


def _spot_image(size, seed):
    """A PSF-like image: a core, rings, and a faint positive background."""
    g = torch.Generator(device='cuda').manual_seed(int(seed))
    y, x = _grid(size)
    d = 0.05 * torch.randn(2, generator=g, dtype=torch.float64, device='cuda')
    r = torch.sqrt((y - d[0]) ** 2 + (x - d[1]) ** 2) * (size / 16)
    img = torch.special.bessel_j1(r + 1e-9) / (r + 1e-9)
    return (img * img + 1e-7 * torch.rand(size, size, generator=g, dtype=torch.float64,
                                          device='cuda')).contiguous()


def prepare(case, seed):
    kind = case['kind']
    s = {'case': case, 'kind': kind}
    if kind == 'dft2':
        s['f'] = _fields(case, seed) if case['count'] > 1 else _fields(case, seed)[0]
        s['alpha'], s['shift'], s['offset'] = _geometry(case, 7)     # one geometry, new fields
    elif kind == 'propagate':
        s['amp'] = _disc(case['npix']).cpu().numpy()
        s['opd'] = _opd(case['npix'], seed).cpu().numpy()
    elif kind == 'fft':
        s['pupil'] = lg.Pupil(amplitude=_disc(case['npix']), opd=_opd(case['npix'], seed),
                              pixelscale=1 / case['npix'], focal_length=FOCAL)
    elif kind == 'gradient':
        s['amp'] = _disc(case['npix'])
        s['opd'] = _opd(case['npix'], seed).requires_grad_(True)
        s['grad'] = _disc(2 * case['det'])
        s['g'] = autodiff.geometry(s['amp'], case['wavelength'], 1 / case['npix'], FOCAL, DU,
                                   shape=case['det'], oversample=2, precision='fp64')
    elif kind == 'retrieval':
        amp, basis, div, targets, c = _retrieval(case, seed)
        s['g'] = autodiff.geometry(amp, case['wavelength'], 1 / case['npix'], FOCAL, DU,
                                   shape=case['det'], oversample=2, precision='split')
        s['pr'] = autodiff.PhaseRetrieval(amp, basis, div, targets, s['g'])
        s['coeffs'] = c.requires_grad_(True)
    elif kind in ('broadband', 'broadband_call'):
        npix = case['npix']
        s['amp'], s['opd'] = _segments(npix), _opd(npix, seed)
        s['lam'], w = _weights(case['waves'])
        if kind == 'broadband_call':
            s['w'] = w
            s['pupil'] = lg.Pupil(amplitude=s['amp'], opd=s['opd'], pixelscale=1 / npix,
                                  focal_length=FOCAL)
            s['pupil'].freeze()
        else:
            rows = (s['amp'] > 0).any(dim=1).nonzero().reshape(-1)
            cols = (s['amp'] > 0).any(dim=0).nonzero().reshape(-1)
            box = (slice(int(rows[0]), int(rows[-1]) + 1), slice(int(cols[0]), int(cols[-1]) + 1))
            geo = plan_geometry((npix, npix), box, [], (1 / npix, 1 / npix), FOCAL, lg.pupil,
                                s['lam'], DU, shape=case['det'], oversample=2)
            s['plan'] = make_plan(geo, precision=case['precision'])
            s['w'] = torch.as_tensor(w, device='cuda').reshape(1, -1)
            s['out'] = torch.empty((1,) + geo.shape_out, dtype=torch.float64, device='cuda')
    elif kind == 'pixelate':
        s['img'] = _spot_image(case['size'], seed)
    return s


def _retrieval(case, seed):
    npix = case['npix']
    g = torch.Generator(device='cuda').manual_seed(int(seed))
    amp = _disc(npix)
    basis = _modes(npix, case['modes'])
    y, x = _grid(npix)
    focus = case['wavelength'] * (y * y + x * x)
    div = [k * focus for k in (-1.0, 0.0, 1.0)]
    t = _disc(2 * case['det'])
    targets = [1e-4 * (k + 1) * t / t.max() for k in range(3)]
    c = 15e-9 * torch.randn(case['modes'], generator=g, dtype=torch.float64, device='cuda')
    return amp, basis, div, targets, c


# --------------------------------------------------------------------- run ---
def run(s):
    case, kind = s['case'], s['kind']
    if kind == 'dft2':
        f = lg.fourier.dft2_batch if case['count'] > 1 else lg.fourier.dft2
        return f(s['f'], s['alpha'], shape=(case['M'], case['N']), shift=s['shift'],
                 offset=s['offset'], precision=case['precision'])
    if kind == 'propagate':
        pupil = lg.Pupil(amplitude=s['amp'], opd=s['opd'], pixelscale=1 / case['npix'],
                         focal_length=FOCAL)
        w = lg.Wavefront(case['wavelength']) * pupil
        return lg.propagate_dft(w, DU, shape=case['det'], oversample=2).intensity
    if kind == 'fft':
        w = lg.Wavefront(case['wavelength']) * s['pupil']
        return lg.propagate_fft(w, DU, oversample=2).field
    if kind == 'gradient':
        img = autodiff.mft_intensity(s['opd'], s['amp'], s['g'])
        grad, = torch.autograd.grad(img, s['opd'], s['grad'])
        return img.detach(), grad
    if kind == 'retrieval':
        loss = s['pr'].loss(s['coeffs'])
        grad, = torch.autograd.grad(loss, s['coeffs'])
        return loss.detach(), grad
    if kind == 'broadband':
        return s['plan'].execute(s['amp'][None], s['opd'][None], s['w'], out=s['out'], check=False)
    if kind == 'broadband_call':
        return lg.broadband_psf(s['pupil'], s['lam'], s['w'], DU, shape=case['det'], oversample=2,
                                precision='fp64')
    return lg.detector.pixelate(s['img'], case['oversample'])


# -------------------------------------------------------------------- work ---
def _mft_flops(m, n, M, N):
    left = M * m * n + M * n * N
    right = m * n * N + M * m * N
    return 8.0 * min(left, right)


def _pupil_dims(case):
    p, M = case['npix'], 2 * case.get('det', 0)
    if case['kind'] in ('broadband', 'broadband_call'):
        return int(0.995 * p), int(0.92 * p), M
    return p, p, M


def work(case):
    kind = case['kind']
    if kind == 'dft2':
        c = case['count']
        return {'bytes': 16 * c * (case['m'] * case['n'] + case['M'] * case['N']),
                'flops': c * _mft_flops(case['m'], case['n'], case['M'], case['N'])}
    if kind == 'pixelate':
        n, o = case['size'], -(-case['size'] // case['oversample'])
        return {'bytes': 8 * (n * n + o * o), 'flops': 20 * n * n * math.log2(n)}
    m, n, M = _pupil_dims(case)
    p = case['npix']
    if kind == 'propagate':
        return {'bytes': 16 * p * p + 8 * M * M, 'flops': _mft_flops(m, n, M, M)}
    if kind == 'fft':
        N = round(p * case['wavelength'] * FOCAL * 2 / DU)
        return {'bytes': 16 * p * p + 16 * N * N, 'flops': 10.0 * N * N * math.log2(N)}
    if kind == 'gradient':
        return {'bytes': 16 * p * p + 16 * M * M + 8 * p * p, 'flops': 2 * _mft_flops(m, n, M, M)}
    if kind == 'retrieval':
        return {'bytes': 8 * p * p * (case['modes'] + 4) + 24 * M * M,
                'flops': 6 * _mft_flops(m, n, M, M) + 4.0 * case['modes'] * p * p}
    return {'bytes': 16 * p * p + 8 * M * M, 'flops': case['waves'] * _mft_flops(m, n, M, M)}


# ------------------------------------------------------------------- exact ---
def _matrix(count_in, count_out, alpha, shift, offset):
    """exp(-2 pi i alpha (r + offset)(u - shift)), [out, in], the cycles taken
    modulo one: alpha is cut into a 20-bit head, whose products are exact, and
    a small rest."""
    r = torch.arange(count_in, dtype=torch.float64, device='cuda') - count_in // 2 + offset
    u = torch.arange(count_out, dtype=torch.float64, device='cuda') - count_out // 2 - shift
    p = u[:, None] * r[None, :]
    m, e = math.frexp(alpha)
    head = math.ldexp(round(math.ldexp(m, 20)), e - 20)
    cycles = torch.remainder(head * p, 1.0) + (alpha - head) * p
    ph = -2 * math.pi * cycles
    return torch.complex(torch.cos(ph), torch.sin(ph))


def _transform(f, alpha, shape, shift=(0.0, 0.0), offset=(0, 0)):
    e1 = _matrix(f.shape[-2], shape[0], alpha[0], shift[0], offset[0])
    e2 = _matrix(f.shape[-1], shape[1], alpha[1], shift[1], offset[1])
    return math.sqrt(abs(alpha[0] * alpha[1])) * (e1 @ f @ e2.transpose(0, 1))


def _alpha(npix, lam):
    a = ((1 / npix) * DU) / (lam * FOCAL * 2)
    return a, a


def _phasor(amp, opd, lam):
    return torch.polar(amp.expand_as(opd).contiguous(), 2 * math.pi * (opd / lam))


def _exact_fft(case, seed):
    p, lam = case['npix'], case['wavelength']
    f = _phasor(_disc(p), _opd(p, seed), lam)
    N = int(np.round(1 / (((1 / p) * DU) / (FOCAL * lam * 2))))
    full = torch.zeros(N, N, dtype=torch.complex128, device='cuda')
    at = (N - p) // 2
    full[at:at + p, at:at + p] = f
    return torch.fft.ifftshift(torch.fft.fft2(torch.fft.fftshift(full), norm='ortho'))


def _exact_gradient(case, seed):
    p, lam = case['npix'], case['wavelength']
    amp, opd, up = _disc(p), _opd(p, seed).requires_grad_(True), _disc(2 * case['det'])
    M = 2 * case['det']
    img = _transform(_phasor(amp, opd, lam), _alpha(p, lam), (M, M)).abs().square()
    grad, = torch.autograd.grad(img, opd, up)
    return img.detach(), grad


def _exact_retrieval(case, seed):
    p, lam, M = case['npix'], case['wavelength'], 2 * case['det']
    amp, basis, div, targets, c = _retrieval(case, seed)
    c = c.requires_grad_(True)
    opd = torch.einsum('k,khw->hw', c, basis)[None] + torch.stack(div)
    img = _transform(_phasor(amp, opd, lam), _alpha(p, lam), (M, M)).abs().square()
    loss = ((img - torch.stack(targets)) ** 2).sum()
    grad, = torch.autograd.grad(loss, c)
    return loss.detach(), grad


def _exact_broadband(case, seed):
    p, M = case['npix'], 2 * case['det']
    amp, opd = _segments(p), _opd(p, seed)
    lam, w = _weights(case['waves'])
    img = torch.zeros(M, M, dtype=torch.float64, device='cuda')
    for k in range(case['waves']):
        F = _transform(_phasor(amp, opd, float(lam[k])), _alpha(p, float(lam[k])), (M, M))
        img += float(w[k]) * F.abs().square()
    return img[None] if case['kind'] == 'broadband' else img


def _spline_matrix(n, x):
    """Rows that take n samples to their cubic spline at x: 12 edge copies a
    side, the spline interpolating with a half-sample-symmetric boundary."""
    pad = 12
    L = n + 2 * pad
    B = np.diag(np.full(L, 4 / 6)) + np.diag(np.full(L - 1, 1 / 6), 1) + np.diag(np.full(L - 1, 1 / 6), -1)
    B[0, 0] += 1 / 6
    B[-1, -1] += 1 / 6
    W = np.zeros((len(x), L))
    for k, xp in enumerate(x + pad):
        for j in range(int(np.floor(xp)) - 1, int(np.floor(xp)) + 3):
            t = abs(xp - j)
            wt = 2 / 3 - t * t + t ** 3 / 2 if t < 1 else max(0.0, 2 - t) ** 3 / 6
            W[k, min(max(j, 0), L - 1)] += wt
    P = np.zeros((L, n))
    P[np.arange(L), np.clip(np.arange(L) - pad, 0, n - 1)] = 1
    return W @ np.linalg.solve(B, P)


def _exact_pixelate(case, seed):
    n, o = case['size'], case['oversample']
    img = _spot_image(n, seed).cpu().numpy()
    k = np.sinc(np.fft.fftfreq(n) * o)
    p = np.abs(np.fft.ifft2(np.fft.fft2(img) * k[:, None] * k[None, :]))
    S = int(np.ceil(n * (1 / o)))
    x = (np.arange(S) - S / 2) / (1 / o) + n / 2
    G = _spline_matrix(n, x)
    out = G @ p @ G.T
    return out * (p.sum() / out.sum())           # the image is positive: nothing is masked


def exact(case, seed):
    kind = case['kind']
    if kind == 'dft2':
        f = _fields(case, seed)
        alpha, shift, offset = _geometry(case, 7)
        F = _transform(f, alpha, (case['M'], case['N']), shift, offset)
        return F if case['count'] > 1 else F[0]
    if kind == 'propagate':
        p, lam, M = case['npix'], case['wavelength'], 2 * case['det']
        f = _phasor(_disc(p), _opd(p, seed), lam)
        return _transform(f, _alpha(p, lam), (M, M)).abs().square().cpu().numpy()
    return {'fft': _exact_fft, 'gradient': _exact_gradient, 'retrieval': _exact_retrieval,
            'broadband': _exact_broadband, 'broadband_call': _exact_broadband,
            'pixelate': _exact_pixelate}[kind](case, seed)
