"""The DFT forms' tile products at the edges of their tiles, K steps and clusters, against numpy in FP64: single rows and
columns, sizes one off a multiple of the 64 x 64 and 32 x 32 tiles, K below one step and with a ragged last step, every
field kind, bands wider than one tile, one and several partial sums."""
import numpy as np
import pytest
import torch

from tests.fixtures import rel_err

pytestmark = pytest.mark.gpu

# FP32 sums of up to ~1000 terms of one magnitude, twice over: a few 1e-7 of the largest value
TOL = 3e-6


@pytest.mark.parametrize('kind', ['f32', 'u8', 'c64'])
@pytest.mark.parametrize('batch,ny,nx,band', [
    (1, 1, 1, (0, 1, 0, 1)),
    (2, 15, 17, (-2, 5, -3, 7)),
    (3, 63, 65, (-16, 33, -31, 63)),
    (1, 130, 250, (-30, 59, -32, 65)),
    (2, 500, 333, (-65, 131, -64, 129)),
    (9, 129, 1000, (-29, 59, -30, 59)),
    (2, 70, 130, (-5, 11, -2, 30)),       # columns up to 27: most of the half are the mirrors of none
    (2, 70, 130, (-5, 11, -27, 28)),      # 0 is the band's end: every other column is a mirror
    (2, 70, 130, (-5, 11, 3, 20)),        # without frequency 0: the general product
    (200, 20, 100, (-3, 7, -31, 64)),
])
def test_band_spectrum(kind, batch, ny, nx, band):
    from opticalimaging_b200 import engine as eng, _native as N
    b = eng.Band(*band)
    dev = torch.device('cuda')
    plan = eng.Plan(ny, nx, b, dev)
    rng = np.random.default_rng(ny + nx)
    nch = 1
    if kind == 'c64':
        nch = 3
        h = rng.standard_normal((batch, ny, nx, nch)) + 1j * rng.standard_normal((batch, ny, nx, nch))
        md, code = torch.from_numpy(h).to(dev, torch.complex64), N.FIELD_COMPLEX_C64
    elif kind == 'u8':
        h = rng.integers(0, 2, (batch, ny, nx)).astype(np.uint8)
        md, code = torch.from_numpy(h).to(dev), N.FIELD_U8
    else:
        h = rng.standard_normal((batch, ny, nx))
        md, code = torch.from_numpy(h).to(dev, torch.float32), N.FIELD_REAL_F32
    got = eng.band_spectrum(md, code, plan, nch=nch, form='dft').cpu().numpy()
    full = np.fft.ifft2(h.reshape(batch, ny, nx, nch).astype(np.complex128), axes=(1, 2)).transpose(0, 3, 1, 2)
    rows, cols = np.arange(b.m0r, b.m0r + b.br) % ny, np.arange(b.m0c, b.m0c + b.bc) % nx
    assert rel_err(got, full[:, :, rows][:, :, :, cols]) < TOL


@pytest.mark.parametrize('count,ny,nx,br,bc', [(1, 1, 1, 1, 1), (1, 3, 257, 2, 3), (2, 17, 512, 9, 8), (1, 66, 513, 30, 65),
                                               (40, 65, 300, 31, 31), (3, 1000, 750, 59, 59), (1, 700, 1500, 117, 260)])
def test_spectrum_to_image(count, ny, nx, br, bc):
    """Image rows and columns around the blocks of 4, 8 and 16 rows and of 256 and 512 columns, odd and even bands."""
    from opticalimaging_b200 import engine as eng, _native as N
    rng = np.random.default_rng(ny * nx)
    ih = rng.standard_normal((count, 2 * br - 1, bc)) + 1j * rng.standard_normal((count, 2 * br - 1, bc))
    dev = torch.device('cuda')
    t = lambda *a: eng.twiddle(*a, device=dev)  # noqa: E731
    sy, sx = t(ny, 2 * br - 1, 0, -(br - 1), ny, -1), t(bc, nx, 0, 0, nx, -1)
    out = torch.full((count, ny, nx), 9.0, device=dev)
    ihd = torch.from_numpy(ih).to(dev, torch.complex64)
    N.call('oi_spectrum_to_image', N.ptr(ihd), count, br, bc, N.ptr(sy), N.ptr(sx), ny, nx, N.ptr(out), N.stream_handle())
    ey = np.exp(-2j * np.pi * np.outer(np.arange(ny), np.arange(-(br - 1), br)) / ny)
    ex = np.exp(-2j * np.pi * np.outer(np.arange(bc), np.arange(nx)) / nx)
    want = (ey @ ih.astype(np.complex64).astype(np.complex128) @ ex).real
    assert rel_err(out.cpu().numpy(), want) < TOL


@pytest.mark.parametrize('nx', [1, 2, 3, 254, 255, 256, 510, 511, 766, 767, 768, 1022, 1024, 1534, 2048])
@pytest.mark.parametrize('count,ny', [(1, 5), (150, 9), (150, 17)])
def test_mirrored_columns(nx, count, ny):
    """Columns x and nx - x from one product: halves around one to nine groups of 128, rows around half blocks."""
    from opticalimaging_b200 import engine as eng, _native as N
    rng = np.random.default_rng(nx + ny)
    br, bc = 3, min(9, (nx + 1) // 2)
    ih = (rng.standard_normal((count, 2 * br - 1, bc)) + 1j * rng.standard_normal((count, 2 * br - 1, bc))).astype(np.complex64)
    dev = torch.device('cuda')
    t = lambda *a: eng.twiddle(*a, device=dev)  # noqa: E731
    sy, sx = t(ny, 2 * br - 1, 0, -(br - 1), ny, -1), t(bc, nx, 0, 0, nx, -1)
    out = torch.full((count, ny, nx), 9.0, device=dev)
    ihd = torch.from_numpy(ih).to(dev)
    N.call('oi_spectrum_to_image', N.ptr(ihd), count, br, bc, N.ptr(sy), N.ptr(sx), ny, nx, N.ptr(out), N.stream_handle())
    ey = np.exp(-2j * np.pi * np.outer(np.arange(ny), np.arange(-(br - 1), br)) / ny)
    ex = np.exp(-2j * np.pi * np.outer(np.arange(bc), np.arange(nx)) / nx)
    assert rel_err(out.cpu().numpy(), (ey @ ih.astype(np.complex128) @ ex).real) < TOL


@pytest.mark.parametrize('nparts', [1, 2, 5])
@pytest.mark.parametrize('count,m,b,ny,nx', [(1, 64, 5, 9, 11), (1, 64, 31, 70, 90), (2, 128, 59, 300, 257), (1, 192, 90, 201, 400),
                                             (20, 128, 64, 131, 150)])
def test_coarse_to_image_dft(nparts, count, m, b, ny, nx):
    """Coarse intensities in partial sums to images: the spectrum in the output's room where it fits (all but 9 x 11)."""
    from opticalimaging_b200 import engine as eng, _native as N
    rng = np.random.default_rng(m + nparts)
    band = eng.Band(-(b // 2), b, -(b // 2), b)
    dev = torch.device('cuda')
    plan = eng.Plan(ny, nx, eng.Band(0, b, 0, b), dev, coarse=(m, m))
    parts = rng.random((nparts, count, m, m))
    c = torch.from_numpy(parts).to(dev, torch.float32)
    ihat = torch.empty(count * (2 * b - 1) * b, dtype=torch.complex64, device=dev)
    out = torch.empty((count, ny, nx), device=dev)
    N.call('oi_coarse_to_image', N.ptr(c), nparts, count, m, m, b, b, N.ptr(plan.gc), N.ptr(plan.gr), N.ptr(plan.sy),
           N.ptr(plan.sx), ny, nx, N.ptr(ihat), N.ptr(out), N.stream_handle())
    q = np.arange(-(b - 1), b)
    s = np.arange(m)
    e = np.exp(2j * np.pi * np.outer(q, s) / m)
    spec = e @ parts.astype(np.float32).astype(np.float64).sum(axis=0) @ e.T / m ** 2      # [count, qr, qc]
    ey = np.exp(-2j * np.pi * np.outer(np.arange(ny), q) / ny)
    ex = np.exp(-2j * np.pi * np.outer(q, np.arange(nx)) / nx)
    want = (ey @ spec @ ex).real
    assert band.br == b and rel_err(out.cpu().numpy(), want) < TOL


def test_coarse_to_image_odd_out():
    """Images that start at an odd float of their buffer: no room for the spectrum's pairs there, same values."""
    from opticalimaging_b200 import engine as eng, _native as N
    dev = torch.device('cuda')
    m, b, ny, nx = 64, 20, 70, 90
    plan = eng.Plan(ny, nx, eng.Band(0, b, 0, b), dev, coarse=(m, m))
    parts = torch.rand((3, 2, m, m), generator=torch.Generator().manual_seed(1)).to(dev)
    ihat = torch.empty(2 * (2 * b - 1) * b, dtype=torch.complex64, device=dev)
    images = []
    for shift in (0, 1):
        c, buf = parts.clone(), torch.empty(2 * ny * nx + 1, device=dev)
        out = buf[shift:shift + 2 * ny * nx]
        N.call('oi_coarse_to_image', N.ptr(c), 3, 2, m, m, b, b, N.ptr(plan.gc), N.ptr(plan.gr), N.ptr(plan.sy),
               N.ptr(plan.sx), ny, nx, N.ptr(ihat), N.ptr(out), N.stream_handle())
        images.append(out.cpu().numpy())
    assert rel_err(images[1], images[0]) < TOL
