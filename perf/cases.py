"""Performance cases of the imaging engine: what a program that uses it has it do, through its public entry points.

    listed()             the cases, from one 256 x 256 clip to 64 clips of 1024 x 1024
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the state a program holds before the call: masks of that seed, and the resident model
    run(state)           one pass through the public entry points, and its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the same outputs in 64 bits, evaluated with plain torch on full-grid transforms

A case has a `task`:
    image    CoherentModel.image on a batch of masks on the device (SOCS kernels or Abbe pupils kept resident)
    ilt      one mask-optimisation gradient: ilt.ilt_loss on sigmoid(logits) and its backward pass
    smo      one source-mask gradient on an Abbe model, as ilt.optimize_source_mask takes it in each iteration
    call     CalculateAerialImage_SOCS: host ScatterField in, host image out, kernels kept
    hopkins  CalculateHopkinsImage: optics and host ScatterField in, host image out, nothing kept
    setup    CalculateTCCMatrix, DecomposeTCC_SOCS and the first image from its kernels
Optics are the package's own benchmark configurations (immersion-mapped NA 1.35 / 193 nm); masks are seeded random
rectangles at about 35 % fill, or, for `c64`, a thin near field in three complex channels.
"""
import math

import numpy as np
import torch

from opticalimaging_b200 import ilt, imaging
from opticalimaging_b200.params import Numerics, Projection, Scatter, Source

WAVELENGTH, NA = 193.0 / 1.44, 1.35 / 1.44     # immersion-mapped: index 1, magnification 1

# Illuminations: shape, points per axis, sigma in / out, vector imaging
SOURCES = {
    'annular-scalar': ('annular', 21, 0.6, 0.9, False),
    'quasar-vector': ('quasar', 31, 0.5, 0.85, True),
    'annular-vector': ('annular', 41, 0.7, 0.95, True),
}
FOCUS = {1: (0.0,), 3: (-40.0, 0.0, 40.0), 5: (-60.0, -30.0, 0.0, 30.0, 60.0)}
RESIST = (30.0, 0.25)                          # steepness and threshold of the sigmoid resist


def _case(name, task, source, period, ny, nx, batch, kernels=0, planes=1, form='default', mask='f32', zernike=False):
    c = {'task': task, 'source': source, 'period': period, 'ny': ny, 'nx': nx, 'batch': batch, 'kernels': kernels,
         'planes': planes, 'form': form, 'mask': mask, 'zernike': zernike}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one clip at a time through a resident scalar Abbe model: an interactive call, all latency
        _case('abbe_256_one', 'image', 'annular-scalar', 1024, 256, 256, 1),
        # the benchmark step: a batch of clips through resident SOCS kernels in the split form
        _case('socs24_1024_64_split', 'image', 'annular-vector', 2048, 1024, 1024, 64, 24, form='bf16x3'),
        # the same kernels in the default FP32 form, a smaller batch
        _case('socs24_1024_8', 'image', 'annular-vector', 2048, 1024, 1024, 8, 24),
        # large clips, whose band is past the split form's range
        _case('socs24_2048_4', 'image', 'annular-vector', 4096, 2048, 2048, 4, 24),
        # a process window as it is served: aberrated vector Abbe, five focus planes, binary masks, split form
        _case('abbe_512_5z_4_split', 'image', 'quasar-vector', 2048, 512, 512, 4, planes=5, form='bf16x3', mask='u8',
              zernike=True),
        # a layout window that is not a power of two
        _case('socs24_1000x750_4', 'image', 'annular-vector', 2048, 1000, 750, 4, 24),
        # thick-mask near fields: three complex channels
        _case('near_field_512_2', 'image', 'annular-vector', 2048, 512, 512, 2, 24, mask='c64'),
        # one iteration's gradient of pixel-based inverse lithography
        _case('ilt_1024_8', 'ilt', 'annular-vector', 2048, 1024, 1024, 8, 16),
        # one iteration's gradients of source-mask optimisation
        _case('smo_256_2', 'smo', 'annular-scalar', 1024, 256, 256, 2),
        # the reference-compatible SOCS call: a pageable host field per call
        _case('call_socs24_1024', 'call', 'annular-vector', 2048, 1024, 1024, 1, 24),
        # the reference-compatible Hopkins call: every call with new optics
        _case('hopkins_call_256', 'hopkins', 'annular-vector', 1024, 256, 256, 1, 16),
        # new optics for many clips: the TCC, its kernels and a first image
        _case('setup_2048nm_512', 'setup', 'annular-vector', 2048, 512, 512, 1, 24),
    ]


# Kernel counts whose cut falls in a gap of the TCC spectrum (a cut between equal eigenvalues has no defined image)
KERNELS = {1024: (8, 16, 24), 2048: (8, 16, 24), 4096: (8, 24)}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('socs', 'socs', 'socs', 'abbe', 'abbe', 'any', 'any', 'near', 'ilt', 'ilt', 'smo', 'call',
                       'hopkins', 'setup'))
    period = rng.choice((1024, 2048))
    k = rng.choice(KERNELS[period])
    side = lambda cap: rng.choice([n for n in (256, 512, 1024, 2048) if n <= cap])  # noqa: E731
    if kind == 'socs':
        ny, nx = side(2048), side(2048)
        if rng.random() < 0.2:
            ny = nx = 2048
            period, k = 4096, 24
        form = 'default' if period == 4096 else rng.choice(('default', 'bf16x3'))
        most = (4 << 22 if period == 4096 else 64 << 20) // (ny * nx)
        return _case('', 'image', 'annular-vector', period, ny, nx, _log(rng, 1, min(64, most)), k, form=form,
                     planes=1 if period == 4096 else rng.choice((1, 1, 3)), mask=rng.choice(('f32', 'u8')))
    if kind == 'abbe':
        n = side(1024)
        source = rng.choice(('annular-scalar', 'quasar-vector'))
        planes = 1 if source == 'annular-scalar' else rng.choice((1, 3, 5))
        return _case('', 'image', source, period, n, n, _log(rng, 1, 4), planes=planes, mask=rng.choice(('f32', 'u8')),
                     form=rng.choice(('default', 'bf16x3')), zernike=source != 'annular-scalar' and rng.random() < 0.5)
    if kind == 'any':   # any grid that holds the band
        return _case('', 'image', 'annular-vector', period, _log(rng, 130, 1400), _log(rng, 130, 1400),
                     _log(rng, 1, 4), k, form='default', mask=rng.choice(('f32', 'u8')))
    if kind == 'near':
        n = side(1024)
        return _case('', 'image', 'annular-vector', period, n, rng.choice((n, _log(rng, 200, 1000))), _log(rng, 1, 2),
                     k, mask='c64')
    if kind == 'ilt':
        ny, nx = side(1024), side(1024)
        return _case('', 'ilt', 'annular-vector', period, ny, nx, _log(rng, 1, 8), k)
    if kind == 'smo':
        n = side(512)
        return _case('', 'smo', rng.choice(('annular-scalar', 'quasar-vector')), period, n, n, _log(rng, 1, 2))
    if kind == 'call':
        n = rng.choice((256, 512, 1024, _log(rng, 200, 1000)))
        return _case('', 'call', 'annular-vector', period, n, n, 1, k, mask=rng.choice(('f32', 'c64')))
    n = rng.choice((256, 512, 1024, _log(rng, 200, 800)))
    return _case('', kind, 'annular-vector', period, n, n, 1, k)


# ------------------------------------------------------------------------------------------------ inputs
def _zernike(case):
    z = np.zeros(37)
    if case['zernike']:
        z[4:] = 0.01 * np.random.default_rng(1002).standard_normal(33)
    return np.float32(z)


def _optics(case):
    shape, points, si, so, vector = SOURCES[case['source']]
    sr, po, nm = Source(), Projection(), Numerics()
    sr.Shape, sr.PntNum, sr.SigmaIn, sr.SigmaOut, sr.OpenAngle = shape, points, si, so, math.pi / 6
    sr.Wavelength, sr.PolarizationVector = WAVELENGTH, [1.0, 0.0]
    po.NA, po.IndexImage, po.Magnification = NA, 1.0, 1.0
    po.FocusRange = torch.tensor(FOCUS[case['planes']])
    po.Aberration_Zernike = torch.from_numpy(_zernike(case))
    nm.ImageCalculationMode = 'vector' if vector else 'scalar'
    nm.ImageCalculationMethod = 'hopkins' if case['kernels'] else 'abbe'
    nm.Hopkins_SettingType, nm.Hopkins_Order = 'order', case['kernels']
    return sr, po, nm


def _rectangles(batch, ny, nx, period, rng, fill=0.35):
    """Binary masks [batch, ny, nx] float32 on the device: rectangles of 30 to 400 nm to about `fill`."""
    count = max(2, round(-math.log(1 - fill) * period ** 2 / 215.0 ** 2))
    w, h = rng.uniform(30.0, 400.0, (2, batch, count))
    x0, y0 = rng.uniform(-200.0, period, (2, batch, count))
    y = torch.from_numpy((np.arange(ny) + 0.5) * period / ny).cuda()
    x = torch.from_numpy((np.arange(nx) + 0.5) * period / nx).cuda()
    w, h, x0, y0 = (torch.from_numpy(a).cuda()[..., None] for a in (w, h, x0, y0))
    rows = ((y >= y0) & (y < y0 + h)).float()
    cols = ((x >= x0) & (x < x0 + w)).float()
    return (torch.bmm(rows.transpose(1, 2), cols) > 0.5).float()


def _inputs(case, seed):
    """The masks of a case: float32 or uint8 [B, ny, nx], complex64 [B, ny, nx, 3], or (logits, target) float32."""
    rng = np.random.default_rng([seed, 71])
    b, ny, nx = case['batch'], case['ny'], case['nx']
    m = _rectangles(b, ny, nx, case['period'], rng)
    if case['task'] in ('ilt', 'smo'):
        g = torch.Generator(device='cuda').manual_seed(seed)
        noise = torch.randn((b, ny, nx), generator=g, device='cuda')
        return 3.0 * (m - 0.5) + 0.5 * noise, m
    if case['mask'] == 'u8':
        return m.to(torch.uint8)
    if case['mask'] == 'c64':   # a near field: the co-polarised channel and weaker cross terms at the edges
        edge = (m - torch.roll(m, 1, 2)) + 1j * (m - torch.roll(m, 1, 1))
        return torch.stack((m * (1 + 0.05j) + 0.1 * edge, 0.08 * edge, 0.05j * torch.roll(edge, 1, 1)),
                           3).to(torch.complex64).contiguous()
    return m


def _field(case, seed):
    """A drop-in caller's ScatterField: complex64 [ny, nx, 3] in pageable host memory."""
    m = _inputs(case, seed)[0]
    if m.dim() == 2:
        m = torch.stack((m, 0 * m, 0 * m), 2).to(torch.complex64)
    return m.cpu()


_MODELS = {}   # the models a program keeps for its optics; masks come and go


def _model(case):
    key = tuple(case[k] for k in ('task', 'source', 'period', 'ny', 'nx', 'kernels', 'planes', 'zernike'))
    if key not in _MODELS:
        sr, po, nm = _optics(case)
        build = imaging.socs_model if case['kernels'] else imaging.abbe_model
        _MODELS[key] = build(sr, po, nm, case['period'], case['period'], case['ny'], case['nx'])
    return _MODELS[key]


def _kernels(case):
    """The full-grid kernels a drop-in caller keeps: [ny, nx, K] on the device."""
    key = ('full',) + tuple(case[k] for k in ('source', 'period', 'ny', 'nx', 'kernels'))
    if key not in _MODELS:
        sr, po, nm = _optics(case)
        tcc, fg = imaging.CalculateTCCMatrix(sr, [case['period']] * 2, po, 0.0, nm)
        _MODELS[key] = imaging.DecomposeTCC_SOCS(tcc, fg, [case['nx'], case['ny']], nm)
    return _MODELS[key]


def prepare(case, seed):
    task = case['task']
    st = {'case': case, 'task': task}
    if task in ('call', 'hopkins', 'setup'):
        sc = Scatter()
        sc.Period_X = sc.Period_Y = case['period']
        sc.ScatterField = _field(case, seed)
        st['source'], st['projection'], st['numerics'] = _optics(case)
        st['scatter'] = sc
        if task == 'call':
            st['kernels'] = _kernels(case)
        return st
    st['model'] = _model(case)
    if task == 'image':
        st['masks'] = _inputs(case, seed)
        st['form'] = None if case['form'] == 'default' else case['form']
        st['channels'] = 3 if case['mask'] == 'c64' else 1
        return st
    logits, st['target'] = _inputs(case, seed)
    st['logits'] = logits.requires_grad_(True)
    st['resist'] = ilt.ResistModel(*RESIST)
    if task == 'smo':
        v = st['model'].weights.shape[1] // (3 if SOURCES[case['source']][4] else 1)
        st['values'] = torch.from_numpy(0.5 + np.random.default_rng([seed, 5]).random(v)).cuda()
    return st


def run(state):
    task = state['task']
    if task == 'image':
        return state['model'].image(state['masks'], nch=state['channels'], form=state['form'])
    if task in ('ilt', 'smo'):
        model, logits = state['model'], state['logits']
        if task == 'smo':
            ilt.set_source_weights(model, state['values'], 1.0)
        logits.grad = None
        mask = torch.sigmoid(logits)
        loss, image = ilt.ilt_loss(model, mask, state['target'], state['resist'])
        if task == 'ilt':
            loss.backward()
            return {'loss': loss.detach(), 'image': image.detach(), 'gradient': logits.grad}
        image.retain_grad()
        loss.backward()
        gv = ilt.source_weight_gradient(model, mask.detach(), image.grad, state['values'], 1.0)
        return {'loss': loss.detach(), 'image': image.detach(), 'gradient': logits.grad, 'source_gradient': gv}
    sr, po, nm, sc = state['source'], state['projection'], state['numerics'], state['scatter']
    if task == 'call':
        image, pupil = imaging.CalculateAerialImage_SOCS(sc, state['kernels'], sr, po)
        return {'image': image, 'pupil': pupil}
    if task == 'hopkins':
        data, pupil = imaging.CalculateHopkinsImage(sr, sc, po, nm)
        return {'image': data.Intensity, 'pupil': pupil}
    ny, nx = sc.ScatterField.shape[:2]
    tcc, fg = imaging.CalculateTCCMatrix(sr, [sc.Period_Y, sc.Period_X], po, 0.0, nm)
    kernels = imaging.DecomposeTCC_SOCS(tcc, fg, [nx, ny], nm)
    image, _ = imaging.CalculateAerialImage_SOCS(sc, kernels, sr, po)
    return {'tcc': tcc, 'image': image}


# --------------------------------------------------------------------------------------------- the least work
def _band(case):
    return 2 * math.ceil(2 * case['period'] * NA / WAVELENGTH) + 1


def _points(case):
    return _source(case)[0].size


def work(case):
    b, z, n, band = case['batch'], case['planes'], case['ny'] * case['nx'], _band(case)
    points, vector = _points(case), SOURCES[case['source']][4]
    fields = case['kernels'] or points * (3 if vector else 1)
    channels = 3 if case['mask'] == 'c64' else 1
    host = case['task'] in ('call', 'hopkins', 'setup')
    per_pixel = 24 if host else {'f32': 4, 'u8': 1, 'c64': 24}[case['mask']]
    grid = (2 * band) ** 2                                 # the samples that hold a field's intensity
    line = 2.5 * n * math.log2(n) / 2                      # one real transform along one axis
    image = channels * line * (2 if channels == 3 else 1) + z * (fields * channels * 5 * grid * math.log2(grid) + line)
    flops, moved = b * image, b * n * (per_pixel + 4 * z)
    if case['task'] in ('ilt', 'smo'):
        flops *= 3                                         # the fields again, and back
        moved = b * n * (4 + 4 + 4 + 4)                    # logits and target in, image and gradient out
    if case['task'] in ('hopkins', 'setup'):
        rank = points * (3 if vector else 1)
        fg = band * band
        flops += 8.0 * fg * rank * min(fg, rank) / 2       # the Gram matrix of the pupil factor, or the TCC
    if case['task'] == 'setup':
        flops += 8.0 * (band * band) ** 2 * rank / 2
        moved += 16.0 * (band * band) ** 2
    return {'bytes': float(moved), 'flops': float(flops)}


# ------------------------------------------------------------------------------------------ 64-bit evaluation
def _source(case):
    """Source points (X, Y, value): the rasterisation decides its points in float32."""
    shape, points, si, so, _ = SOURCES[case['source']]
    c = torch.linspace(-1, 1, points)
    X, Y = torch.meshgrid(c, c, indexing='ij')
    r = torch.sqrt(X.pow(2) + Y.pow(2))
    keep = (r <= so) & (r >= si)
    value = 1.0 / ((so ** 2 - si ** 2) * math.pi)
    if shape == 'quasar':
        angle = math.pi / 6
        value, half, th = 0.5 / ((so ** 2 - si ** 2) * angle), angle / 2, torch.atan2(Y, X)
        a = torch.abs(th)
        keep &= ((a <= half) | (a >= math.pi - half) | (torch.abs(th - math.pi / 2) <= half)
                 | (torch.abs(th + math.pi / 2) <= half))
    keep &= (X ** 2 + Y ** 2) <= 1
    keep[(points - 1) // 2, (points - 1) // 2] = False
    X, Y = X[keep].numpy(), Y[keep].numpy()
    return X, Y, np.full(X.size, np.float32(value))


def _aberration(z, rho, theta):
    """Fringe Zernike phase in waves: group g holds n + m = 2 g, m = g .. 0, cosine before sine."""
    out, j = torch.zeros_like(rho), 0
    order = [(2 * g - m, m, s) for g in range(6) for m in range(g, -1, -1) for s in ((0,) if m == 0 else (1, -1))]
    for j, (n, m, s) in enumerate(order + [(12, 0, 0)]):
        if z[j] == 0:
            continue
        radial = sum((-1) ** k * math.factorial(n - k) / (math.factorial(k) * math.factorial((n + m) // 2 - k)
                     * math.factorial((n - m) // 2 - k)) * rho ** (n - 2 * k) for k in range((n - m) // 2 + 1))
        out = out + float(z[j]) * radial * (1 if s == 0 else torch.cos(m * theta) if s > 0 else torch.sin(m * theta))
    return out


def _pupils(case, rows, cols, focus, inside):
    """Pupil of every (point, component) at float32 frequencies rows x cols: [S, E, rows, cols] complex128."""
    X, Y, _ = _source(case)
    dev = 'cuda'
    u = torch.from_numpy(rows).double().to(dev)[None, :, None] + torch.from_numpy(X).double().to(dev)[:, None, None]
    v = torch.from_numpy(cols).double().to(dev)[None, None, :] + torch.from_numpy(Y).double().to(dev)[:, None, None]
    r2 = (u * u + v * v) * inside
    ab = _aberration(_zernike(case), r2.sqrt(), torch.atan2(v.expand_as(r2), u.expand_as(r2)))
    s = (1 - NA ** 2 * r2).clamp_min(0)                    # magnification 1: the obliquity factor is 1
    p = torch.polar(inside.double(), 2 * math.pi * (ab + s.sqrt() * focus / WAVELENGTH))
    if not SOURCES[case['source']][4]:
        return p[:, None]
    a, b = (NA * u).expand_as(r2) * inside, (NA * v).expand_as(r2) * inside
    gam = (1 - a * a - b * b).clamp_min(0).sqrt()
    return torch.stack(((1 - a * a / (1 + gam)) * p, (-a * b / (1 + gam)) * p, -a * p), 1)


def _abbe_fields(case):
    """(row frequencies, column frequencies, fields [Z][S*E] complex128, weights [S*E]) of the Abbe sum."""
    X, Y, V = _source(case)
    np_ = case['period'] / (WAVELENGTH / NA)
    r = int(math.ceil(2 * np_)) + 2
    m = [np.arange(-min(r, n // 2), min(r, (n + 1) // 2 - 1) + 1) for n in (case['ny'], case['nx'])]
    f = [np.float32(1 / np_) * k.astype(np.float32) for k in m]
    fm, gm = f[0][:, None], f[1][None, :]
    rho2 = (fm * fm + gm * gm)[None] + np.float32(2) * (X[:, None, None] * fm + Y[:, None, None] * gm)
    inside = torch.from_numpy(rho2 + (X * X + Y * Y)[:, None, None] <= 1).cuda()
    planes = [_pupils(case, f[0], f[1], z, inside).flatten(0, 1) for z in FOCUS[case['planes']]]
    w = torch.from_numpy(V).double().cuda()
    return m[0], m[1], planes, (w / w.sum()).repeat_interleave(planes[0].shape[0] // w.numel())


def _tcc_factor(case, focus):
    """(frequencies, h [FG, S*E]) with TCC = h h^H."""
    X, Y, V = _source(case)
    np_ = np.float32(case['period'] / (WAVELENGTH / NA))
    r = int(np.ceil(np.float32(2) * np_))
    m = np.arange(-r, r + 1)
    f = (np.float32(1) / np_) * m.astype(np.float32)
    u, v = f[:, None] + X[:, None, None], f[None, :] + Y[:, None, None]
    inside = torch.from_numpy(np.sqrt(u * u + v * v) <= 1).cuda()
    w = torch.from_numpy(V).double().cuda()
    p = _pupils(case, f, f, focus, inside) * (w / w.sum()).sqrt()[:, None, None, None]
    return m, p.flatten(2).flatten(0, 1).T.contiguous()


def _socs_fields(case):
    """(row frequencies, column frequencies, kernels [Z][K] complex128, weights) of the truncated Hopkins sum."""
    planes = []
    for z in FOCUS[case['planes']]:
        m, h = _tcc_factor(case, z)
        lam, v = torch.linalg.eigh(h.conj().T @ h)
        k = v[:, -case['kernels']:]
        planes.append((h @ k).T.reshape(-1, m.size, m.size))
    # the kernel grid is embedded centred and fftshifted: on odd grids that is one frequency below the centre
    at = [m - m[0] + (n - m.size + 1) // 2 + n // 2 - n for n in (case['ny'], case['nx'])]
    return at[0], at[1], planes, torch.ones(case['kernels'], dtype=torch.float64, device='cuda')


def _fields(case):
    return _socs_fields(case) if case['kernels'] else _abbe_fields(case)


def _embed(p, spec, mr, mc):
    """Full-grid spectra of the fields p [K, br, bc] .* spec [ny, nx] on the band."""
    ir = torch.from_numpy(mr % spec.shape[0]).cuda()[:, None]
    ic = torch.from_numpy(mc % spec.shape[1]).cuda()[None, :]
    full = torch.zeros((p.shape[0],) + spec.shape, dtype=torch.complex128, device='cuda')
    full[:, ir, ic] = p * spec[ir, ic]
    return full


def _chunks(p, w, n):
    step = max(1, (1 << 28) // (16 * n))
    return [(p[i:i + step], w[i:i + step]) for i in range(0, p.shape[0], step)]


def _image(mask, fields):
    """[Z, ny, nx] float64 of one mask [ny, nx] or [ny, nx, C]."""
    mr, mc, planes, w = fields
    chans = [mask] if mask.dim() == 2 else [mask[..., c] for c in range(mask.shape[2])]
    out = []
    for p in planes:
        acc = torch.zeros(mask.shape[:2], dtype=torch.float64, device='cuda')
        for h in chans:
            spec = torch.fft.ifft2(h.to(torch.complex128))
            for pc, wc in _chunks(p, w, spec.numel()):
                e = torch.fft.fft2(_embed(pc, spec, mr, mc))
                acc += torch.einsum('k,kyx->yx', wc, e.real ** 2 + e.imag ** 2)
        out.append(acc)
    return torch.stack(out)


def _gradients(logits, target, fields, values=None):
    """(loss, image [Z, ny, nx], dL/dlogits, dL/dvalues or None) of one clip of one focus plane."""
    mr, mc, planes, w = fields
    p, (a, thr) = planes[0], RESIST
    t = torch.sigmoid(logits.double())
    image = _image(t, fields)
    s = torch.sigmoid(a * (image[0] - thr))
    r = s - target.double()
    g = 2 * r * a * s * (1 - s)
    spec = torch.fft.ifft2(t.to(torch.complex128))
    back, dots = torch.zeros_like(spec), []
    for pc, wc in _chunks(p, w, spec.numel()):
        e = torch.fft.fft2(_embed(pc, spec, mr, mc))
        dots.append((g * (e.real ** 2 + e.imag ** 2)).sum(dim=(1, 2)))
        q = torch.fft.ifft2(g * e)                         # the adjoint of the field's transform, over ny nx
        back += _embed_sum(pc.conj() * wc[:, None, None], q, mr, mc)
    grad = 2 * torch.fft.fft2(back).real * t * (1 - t)
    gv = None
    if values is not None:
        d = torch.cat(dots).view(values.numel(), -1).sum(dim=1)
        gv = (d - (d * values).sum() / values.sum()) / values.sum()
    return (r * r).sum(), image, grad, gv


def _embed_sum(p, q, mr, mc):
    """sum_k p[k] .* q[k] on the band, as a full grid."""
    ir = torch.from_numpy(mr % q.shape[1]).cuda()[:, None]
    ic = torch.from_numpy(mc % q.shape[2]).cuda()[None, :]
    full = torch.zeros(q.shape[1:], dtype=torch.complex128, device='cuda')
    full[ir, ic] = (p * q[:, ir, ic]).sum(dim=0)
    return full


def _pupil_image(case, field):
    """The cropped centred spectrum, NaN outside the unit disc."""
    np_ = case['period'] / (WAVELENGTH / NA)
    ny, nx, _ = field.shape
    h = torch.fft.ifftshift(field.cuda().to(torch.complex128), dim=(0, 1))
    hk = torch.fft.fftshift(torch.fft.ifft2(h, dim=(0, 1)), dim=(0, 1)) * np_ ** 2
    f, g = (np.float32(1 / np_) * np.arange(-(n // 2), (n + 1) // 2).astype(np.float32) for n in (nx, ny))
    hk[torch.from_numpy(g[:, None] ** 2 + f[None, :] ** 2 > 1).cuda()] = float('nan')
    o = int(np_) + 3
    return hk[ny // 2 - o:ny // 2 + o, nx // 2 - o:nx // 2 + o]


def exact(case, seed):
    fields = _fields(case)
    task = case['task']
    if task == 'image':
        masks = _inputs(case, seed)
        out = torch.stack([_image(m, fields) for m in masks])
        return out
    if task in ('ilt', 'smo'):
        logits, target = _inputs(case, seed)
        values = None
        if task == 'smo':
            values = torch.from_numpy(0.5 + np.random.default_rng([seed, 5]).random(_points(case))).cuda()
            mr, mc, planes, w = fields
            fields = mr, mc, planes, (values / values.sum()).repeat_interleave(w.numel() // values.numel())
        got = [_gradients(x, t, fields, values) for x, t in zip(logits, target)]
        out = {'loss': sum(g[0] for g in got), 'image': torch.stack([g[1] for g in got]),
               'gradient': torch.stack([g[2] for g in got])}
        return dict(out, source_gradient=torch.stack([g[3] for g in got])) if task == 'smo' else out
    field = _field(case, seed)
    image = _image(field.cuda(), fields)
    if task == 'setup':
        _, h = _tcc_factor(case, 0.0)
        return {'tcc': h @ h.conj().T, 'image': image[0]}
    return {'image': image[0] if task == 'call' else image, 'pupil': _pupil_image(case, field)}
