"""More images than a grid's second dimension holds (65535)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m', [64, 128, 256])
def test_synthesis_of_many_images(m):
    """oi_coarse_to_image_fft with 65537 images of 256 x 256 (17 GB): each equals the image of the same coarse intensity
    alone."""
    from opticalimaging_b200 import engine as eng, _native as N
    dev, count, br, bc, n = torch.device('cuda'), 65537, 2, 2, 256
    t = lambda *a: eng.twiddle(*a, device=dev)  # noqa: E731
    gc, gr = t(m, bc, 0, 0, m, +1), t(m, 2 * br - 1, 0, -(br - 1), m, +1)
    wm, tn = t(1, m, 1, 0, m, +1), eng.fft_tables(n, dev)

    def images(coarse):
        k = coarse.shape[0]
        ihat = torch.empty(k * (2 * br - 1) * bc, dtype=torch.complex64, device=dev)
        v = torch.empty(k * bc * n, dtype=torch.complex64, device=dev)
        out = torch.full((k, n, n), 9.0, device=dev)
        N.call('oi_coarse_to_image_fft', N.ptr(coarse), 1, k, m, m, br, bc, N.ptr(gc), N.ptr(gr), N.ptr(wm), N.ptr(wm),
               N.ptr(tn), N.ptr(tn), n, n, N.ptr(ihat), N.ptr(v), N.ptr(out), N.stream_handle())
        return out

    seven = torch.rand((7, m, m), generator=torch.Generator().manual_seed(m)).to(dev)
    want = images(seven)
    got = images(seven.repeat(count // 7 + 1, 1, 1)[:count].contiguous())
    for i0 in range(0, count, 7 * 512):
        g = got[i0:i0 + 7 * 512]
        # the few images take row blocks of another size: the same sums, each of a few FP32 operations
        assert float((g - want.repeat(513, 1, 1)[:g.shape[0]]).abs().max()) < 1e-6


def test_hermitian_half_of_many_images():
    from opticalimaging_b200 import _native as N
    B, nz, parts, br, bc = 65537, 2, 3, 3, 2
    rng = np.random.default_rng(1)
    w = (rng.standard_normal((parts, B, nz, br, bc)) + 1j * rng.standard_normal((parts, B, nz, br, bc))).astype(np.complex64)
    wd = torch.from_numpy(w).cuda()
    half = torch.full((B, 3, 2), 9.0, dtype=torch.complex64, device='cuda')
    N.call('oi_hermitian_half', N.ptr(wd), parts, B, nz, -1, br, 0, bc, 1.5, N.ptr(half), N.stream_handle())
    full = np.zeros((B, 3, 3), complex)
    full[:, :, 1:] = w.astype(complex).sum(axis=(0, 2))
    want = (full + np.conj(full[:, ::-1, ::-1]))[:, :, 1:] * 1.5
    want[:, :, 0] *= 0.5
    # sums of 12 FP32 values of a few units
    assert np.max(np.abs(half.cpu().numpy() - want)) < 2e-5
