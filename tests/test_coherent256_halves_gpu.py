"""The 256 x 256 coherent sum with one block per share and with one per half of its columns (chosen by the number of
blocks): the same image either way, and against a direct FP64 evaluation."""
import numpy as np
import pytest
import torch

from tests.fixtures import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('br,bc', [(65, 128), (117, 117), (128, 66)])
@pytest.mark.parametrize('B,Z,K,nsplit', [(1, 1, 1, 1), (1, 2, 5, 3), (80, 1, 2, 1), (75, 2, 1, 1), (149, 1, 1, 1)])
def test_matches_fp64(br, bc, B, Z, K, nsplit):
    from opticalimaging_b200 import engine as eng, _native as N
    dev = torch.device('cuda')
    g = torch.Generator(device='cuda').manual_seed(br + B)
    cplx = lambda *s: torch.randn(s, generator=g, device='cuda', dtype=torch.complex64)  # noqa: E731
    band, pupils, w = cplx(B, 1, br, bc), cplx(Z, K, br, bc), torch.rand((Z, K), generator=g, device='cuda')
    tw = eng.twiddle(1, 256, 1, 0, 256, +1, dev)
    out = torch.full((nsplit, B, Z, 256, 256), 9.0, device=dev)
    N.call('oi_coherent_coarse_fft', N.ptr(band), B, 1, -40, br, -50, bc, N.ptr(pupils), 0, N.ptr(w), Z, K, 256, 256,
           N.ptr(tw), N.ptr(tw), nsplit, N.ptr(out), N.stream_handle())
    got = out.sum(dim=0)
    for b in {0, B // 2, B - 1}:
        for z in range(Z):
            full = torch.zeros((K, 256, 256), dtype=torch.complex128, device=dev)
            full[:, :br, :bc] = pupils[z].to(torch.complex128) * band[b, 0].to(torch.complex128)
            e = torch.fft.fft2(full)
            want = (w[z].double()[:, None, None] * (e.real ** 2 + e.imag ** 2)).sum(dim=0)
            assert rel_err(got[b, z].cpu().numpy(), want.cpu().numpy()) < 5e-6
