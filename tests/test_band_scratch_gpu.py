"""band_spectrum with a caller's scratch that starts at any complex value of its buffer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shift', [0, 1, 2])
def test_complex_fields(shift):
    from opticalimaging_b200 import engine as eng, _native as N
    dev, nch, n = torch.device('cuda'), 3, 256
    plan = eng.Plan.get(n, n, eng.Band(-15, 31, -15, 31), dev)
    g = torch.Generator(device='cuda').manual_seed(5)
    field = torch.randn((2, n, n, nch), generator=g, dtype=torch.complex64, device=dev)
    want = torch.fft.ifft2(field.to(torch.complex128), dim=(1, 2)).permute(0, 3, 1, 2)
    m = torch.arange(-15, 16, device=dev) % n
    want = want[:, :, m][:, :, :, m]
    buf = torch.empty(2 * nch * n * 31 + shift, dtype=torch.complex64, device=dev)
    got = eng.band_spectrum(field, N.FIELD_COMPLEX_C64, plan, nch=nch, scratch=buf[shift:])
    # two FP32 transforms of 256 points
    assert float((got - want).abs().max()) < 3e-6 * float(want.abs().max())
