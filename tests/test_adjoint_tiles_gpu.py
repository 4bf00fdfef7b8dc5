"""The adjoint kernel against a direct FP64 evaluation: bands of 1, odd and even sizes up to 64 per axis, offsets that are
not centred, several fields, channels and planes, more field shares than fields divide into, and the field dots alone."""
import numpy as np
import pytest
import torch

from tests.fixtures import rel_err

pytestmark = pytest.mark.gpu


def _direct(band, pupils, weights, gc, m0r, m0c):
    B, C, br, bc = band.shape
    Z, K = pupils.shape[:2]
    er = np.exp(-2j * np.pi * np.outer(np.arange(128), m0r + np.arange(br)) / 128)
    ec = np.exp(-2j * np.pi * np.outer(m0c + np.arange(bc), np.arange(128)) / 128)
    w = np.zeros((B, C, br, bc), complex)
    dots = np.zeros((B, Z, K * C))
    for b in range(B):
        for z in range(Z):
            for k in range(K):
                for c in range(C):
                    e = er @ (pupils[z, k] * band[b, c]) @ ec
                    dots[b, z, k * C + c] = np.sum(gc[b, z] * np.abs(e) ** 2)
                    f = er.conj().T @ (gc[b, z] * e) @ ec.conj().T
                    w[b, c] += weights[z, k] * np.conj(pupils[z, k]) * f
    return w, dots


@pytest.mark.parametrize('br,bc,m0r,m0c', [(1, 1, 0, 0), (8, 9, -3, 2), (33, 31, -16, -15), (59, 59, -29, -30), (64, 63, -5, -62),
                                           (7, 64, 0, -32)])
@pytest.mark.parametrize('B,C,Z,K', [(1, 1, 1, 1), (2, 1, 2, 5), (1, 3, 1, 4)])
def test_adjoint_matches_fp64(br, bc, m0r, m0c, B, C, Z, K):
    from opticalimaging_b200 import engine as eng, _native as N
    rng = np.random.default_rng(br * bc + K)
    cplx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    band, pupils = cplx(B, C, br, bc), cplx(Z, K, br, bc)
    weights, gc = rng.random((Z, K)), rng.standard_normal((B, Z, 128, 128))
    want, wdots = _direct(band, pupils, weights, gc, m0r, m0c)
    dev = torch.device('cuda')
    d = lambda a, t: torch.from_numpy(a).to(dev, t).contiguous()  # noqa: E731
    bd, pd, wd, gd = d(band, torch.complex64), d(pupils, torch.complex64), d(weights, torch.float32), d(gc, torch.float32)
    tw = eng.twiddle(1, 128, 1, 0, 128, +1, dev)
    for nsplit in {1, min(3, K * C), K * C}:
        w = torch.full((nsplit, B, Z, C, br, bc), 9.0, dtype=torch.complex64, device=dev)
        dots = torch.full((2, B, Z, K * C), 9.0, device=dev)
        N.call('oi_coherent_adjoint', N.ptr(bd), B, C, m0r, br, m0c, bc, N.ptr(pd), N.ptr(wd), Z, K, N.ptr(gd), 128, 128,
               N.ptr(tw), N.ptr(tw), nsplit, N.ptr(w), N.ptr(dots[0]), N.stream_handle())
        N.call('oi_coherent_field_dots', N.ptr(bd), B, C, m0r, br, m0c, bc, N.ptr(pd), N.ptr(wd), Z, K, N.ptr(gd), 128, 128,
               N.ptr(tw), N.ptr(tw), nsplit, N.ptr(dots[1]), N.stream_handle())
        # FP32 transforms of 128 points there and back, and sums of a few fields; the dots sum 16384 values of both signs
        assert rel_err(w.sum(dim=(0, 2)).cpu().numpy(), want) < 3e-6
        for x in dots:
            assert np.max(np.abs(x.cpu().numpy() - wdots)) < 2e-6 * np.max(np.sum(np.abs(gc), axis=(2, 3))) * 4 * br * bc
        assert torch.equal(dots[0], dots[1])


@pytest.mark.parametrize('m0r,br,m0c,bc', [(0, 1, 0, 1), (-3, 5, -1, 9), (-29, 59, -29, 59), (2, 4, -7, 3)])
@pytest.mark.parametrize('nparts,B,Z', [(1, 1, 1), (3, 2, 2)])
def test_hermitian_half(m0r, br, m0c, bc, nparts, B, Z):
    from opticalimaging_b200 import _native as N
    rng = np.random.default_rng(br)
    w = (rng.standard_normal((nparts, B, Z, br, bc)) + 1j * rng.standard_normal((nparts, B, Z, br, bc)))
    R, C = max(abs(m0r), abs(m0r + br - 1)), max(abs(m0c), abs(m0c + bc - 1))
    full = np.zeros((B, 2 * R + 1, 2 * C + 1), complex)
    full[:, m0r + R:m0r + R + br, m0c + C:m0c + C + bc] = w.sum(axis=(0, 2))
    want = (full + np.conj(full[:, ::-1, ::-1]))[:, :, C:] * 1.5
    want[:, :, 0] *= 0.5
    wd = torch.from_numpy(w).cuda().to(torch.complex64)
    half = torch.empty((B, 2 * R + 1, C + 1), dtype=torch.complex64, device='cuda')
    N.call('oi_hermitian_half', N.ptr(wd), nparts, B, Z, m0r, br, m0c, bc, 1.5, N.ptr(half), N.stream_handle())
    assert rel_err(half.cpu().numpy(), want) < 1e-6
