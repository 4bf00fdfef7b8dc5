"""The adjoint's coarse copy of an image gradient at every grid size per axis, the smallest and largest bands of each column
variant (1, 32, 33, 64), and counts on both sides of the rows' rule, against numpy in FP64."""
import numpy as np
import pytest
import torch

from tests.fixtures import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('ny,nx', [(256, 256), (512, 2048), (1024, 512), (2048, 1024)])
@pytest.mark.parametrize('br,bc', [(1, 1), (1, 64), (32, 31), (33, 32), (59, 59), (64, 2), (64, 64)])
@pytest.mark.parametrize('count', [1, 3, 5])
def test_coarse_gradient(ny, nx, br, bc, count):
    from opticalimaging_b200 import engine as eng, _native as N
    rng = np.random.default_rng(ny + br + count)
    g = rng.standard_normal((count, ny, nx)).astype(np.float32)
    dev = torch.device('cuda')
    gd = torch.from_numpy(g).to(dev)
    tab = [eng.fft_tables(n, dev) for n in (nx, ny, 128)] + [eng.twiddle(1, 128, 1, 0, 128, +1, dev)]
    t = torch.empty(count * bc * (ny + 128), dtype=torch.complex64, device=dev)
    out = torch.full((count, 128, 128), 9.0, device=dev)
    scale = 1.0 / (ny * nx)
    N.call('oi_coarse_gradient_fft', N.ptr(gd), count, ny, nx, br, bc, *[N.ptr(x) for x in tab], scale, N.ptr(t), N.ptr(out),
           N.stream_handle())
    q, p, s = np.arange(-(br - 1), br), np.arange(-(bc - 1), bc), np.arange(128)
    e = lambda a, b, n, sg: np.exp(sg * 2j * np.pi * (np.outer(a, b) % n) / n)  # noqa: E731
    ghat = np.fft.ifft2(g.astype(np.float64), axes=(1, 2))[:, q % ny][:, :, p % nx]     # over ny nx already
    want = (e(s, q, 128, -1) @ ghat @ e(p, s, 128, -1)).real
    # FP32 transforms there and back: some 1e-7 of the largest value
    assert rel_err(out.cpu().numpy(), want) < 3e-6
