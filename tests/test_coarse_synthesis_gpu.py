"""The FFT form's synthesis (coarse intensities in partial sums to images) on every coarse grid of 64, 128 and 256 per
axis and every output size, at the smallest and largest bands of each gather (1, 64, 65, 128), against numpy in FP64."""
import numpy as np
import pytest
import torch

from tests.fixtures import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('ny,nx', [(256, 256), (512, 1024), (2048, 512), (1024, 2048)])
@pytest.mark.parametrize('mr,mc,br,bc', [(64, 64, 1, 1), (64, 64, 32, 32), (128, 64, 59, 31), (64, 128, 30, 64),
                                         (128, 128, 64, 59), (256, 256, 65, 128), (256, 128, 117, 33), (128, 256, 2, 117),
                                         (256, 256, 128, 65)])
@pytest.mark.parametrize('count,nparts', [(1, 1), (2, 7), (30, 2)])
def test_coarse_to_image_fft(ny, nx, mr, mc, br, bc, count, nparts):
    from opticalimaging_b200 import engine as eng, _native as N
    if count * ny * nx > 1 << 24:
        count = 3
    rng = np.random.default_rng(mr + br + nparts)
    dev = torch.device('cuda')
    parts = rng.random((nparts, count, mr, mc)).astype(np.float32)
    c = torch.from_numpy(parts).to(dev)
    t = lambda *a: eng.twiddle(*a, device=dev)  # noqa: E731
    gc, gr = t(mc, bc, 0, 0, mc, +1), t(mr, 2 * br - 1, 0, -(br - 1), mr, +1)
    wr, wc = t(1, mr, 1, 0, mr, +1), t(1, mc, 1, 0, mc, +1)
    ty, tx = eng.fft_tables(ny, dev), eng.fft_tables(nx, dev)
    ihat = torch.empty(count * (2 * br - 1) * bc, dtype=torch.complex64, device=dev)
    v = torch.empty(count * bc * ny, dtype=torch.complex64, device=dev)
    out = torch.full((count, ny, nx), 9.0, device=dev)
    N.call('oi_coarse_to_image_fft', N.ptr(c), nparts, count, mr, mc, br, bc, N.ptr(gc), N.ptr(gr), N.ptr(wr), N.ptr(wc),
           N.ptr(ty), N.ptr(tx), ny, nx, N.ptr(ihat), N.ptr(v), N.ptr(out),
           N.stream_handle())
    d64 = torch.complex128
    q, s = torch.arange(-(br - 1), br, device=dev), torch.arange(mr, device=dev)
    p, r = torch.arange(-(bc - 1), bc, device=dev), torch.arange(mc, device=dev)
    e = lambda a, b, n, sg: torch.exp(sg * 2j * torch.pi * (torch.outer(a, b) % n).to(d64) / n)  # noqa: E731
    spec = e(q, s, mr, 1) @ c.double().sum(dim=0).to(d64) @ e(r, p, mc, 1) / (mr * mc)
    y, x = torch.arange(ny, device=dev), torch.arange(nx, device=dev)
    want = (e(y, q, ny, -1) @ spec @ e(p, x, nx, -1)).real
    # FP32 transforms of O(1) values in [0, 1): some 1e-7 of the largest
    assert rel_err(out.cpu().numpy(), want.cpu().numpy()) < 3e-6
