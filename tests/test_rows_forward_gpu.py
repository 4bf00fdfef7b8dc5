"""The FFT form's forward passes on both sides of every outer-sum range (bands reaching 31 / 32, 63 / 64, 127 / 128), for
every row length, real, uint8 and complex fields of one to four channels, against numpy in FP64."""
import numpy as np
import pytest
import torch

from tests.fixtures import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind,nch', [('f32', 1), ('u8', 1), ('c64', 1), ('c64', 3), ('c64', 4)])
@pytest.mark.parametrize('ny,nx', [(256, 256), (256, 512), (512, 1024), (256, 2048)])
@pytest.mark.parametrize('m0c,bc', [(0, 1), (-31, 63), (-32, 64), (-3, 36), (-63, 127), (-64, 10), (0, 65), (-100, 201), (100, 12)])
def test_band_spectrum(kind, nch, ny, nx, m0c, bc):
    from opticalimaging_b200 import engine as eng, _native as N
    if 2 * max(abs(m0c), abs(m0c + bc - 1)) >= nx or 2 * bc - 1 > nx:
        pytest.skip('the band or its intensity passes Nyquist: not an FFT-form plan')
    b = eng.Band(-9, 20, m0c, bc)
    dev = torch.device('cuda')
    plan = eng.Plan(ny, nx, b, dev, coarse=(64, ((2 * bc + 63) // 64) * 64))
    rng = np.random.default_rng(nx + bc)
    batch = 2
    if kind == 'c64':
        h = rng.standard_normal((batch, ny, nx, nch)) + 1j * rng.standard_normal((batch, ny, nx, nch))
        md, code = torch.from_numpy(h).to(dev, torch.complex64), N.FIELD_COMPLEX_C64
    elif kind == 'u8':
        h = rng.integers(0, 2, (batch, ny, nx)).astype(np.uint8)
        md, code = torch.from_numpy(h).to(dev), N.FIELD_U8
    else:
        h = rng.standard_normal((batch, ny, nx))
        md, code = torch.from_numpy(h).to(dev, torch.float32), N.FIELD_REAL_F32
    assert plan.fft
    got = eng.band_spectrum(md, code, plan, nch=nch, form='fft').cpu().numpy()
    full = np.fft.ifft2(h.reshape(batch, ny, nx, nch).astype(np.complex128), axes=(1, 2)).transpose(0, 3, 1, 2)
    rows, cols = np.arange(b.m0r, b.m0r + b.br) % ny, np.arange(b.m0c, b.m0c + b.bc) % nx
    # FP32 transforms of O(1) values: a few 1e-7 of the largest
    assert rel_err(got, full[:, :, rows][:, :, :, cols]) < 3e-6
