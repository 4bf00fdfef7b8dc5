"""The FP64 top-K eigensolver at the edges of its tiles and of its filter: block sizes around the 64-row tiles and the
16-value chunks, fewer independent columns than the block holds, spectra that separate well, badly and not at all."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _spectrum(kind, n):
    i = torch.arange(n, dtype=torch.float64)
    if kind == 'decay':                       # a TCC's: one decade per 12 values
        return torch.exp(-0.19 * i)
    if kind == 'slow':                        # the unwanted interval nearly touches the wanted values
        return 1.0 / (1.0 + 0.05 * i)
    if kind == 'one':                         # every column of the block the same direction
        return torch.where(i < 1, 1.0, 0.0).double()
    return torch.where(i < 20, 1.0 / (1.0 + i), torch.zeros_like(i))    # rank 20


@pytest.mark.parametrize('n', [64, 65, 127, 200, 961, 2400])
@pytest.mark.parametrize('kind', ['decay', 'slow', 'rank', 'one'])
@pytest.mark.parametrize('k', [1, 16, 48])
def test_dense_matches_eigh(n, kind, k):
    from opticalimaging_b200 import imaging as oi
    g = torch.Generator().manual_seed(n)
    A = torch.randn((n, min(n, 200)), generator=g, dtype=torch.complex128)
    U = torch.linalg.qr(A)[0]
    lam = _spectrum(kind, U.shape[1])
    T = ((U * lam) @ U.conj().T).cuda()
    vals, vecs = oi.eig_topk(k, tcc=T)
    lam = lam[:k].cuda()
    # residual of the pairs below the solver's tolerance (1e-13 of lambda_0, and rounding of the product), values as
    # close (Hermitian: |error| <= residual), wanted vectors orthonormal
    r = T @ vecs - vecs * vals
    assert float(r.norm(dim=0).max()) < 2e-13
    assert float((vals - lam).abs().max()) < 2e-13
    live = int((lam > 1e-12).sum())
    v = vecs[:, :live]
    assert float((v.conj().T @ v - torch.eye(live, device='cuda')).abs().max()) < 1e-12


@pytest.mark.parametrize('ne,s', [(1, 1), (1, 17), (3, 64), (3, 70)])
@pytest.mark.parametrize('n', [66, 300])
def test_factored_matches_dense_and_skips_zero_blocks(ne, s, n):
    """T = sum_e h_e h_e^H from h whose samples are zero outside a moving window, as shifted pupils are."""
    from opticalimaging_b200 import imaging as oi
    rng = np.random.default_rng(s)
    h = rng.standard_normal((ne, n, s)) + 1j * rng.standard_normal((ne, n, s))
    row, col = np.arange(n)[:, None] / n, np.arange(s)[None, :] / s
    h = torch.from_numpy(h * (np.abs(row - 0.2 - 0.6 * col) < 0.25)).cuda()
    H = h.permute(1, 0, 2).reshape(n, ne * s)
    k = min(8, ne * s)
    vals, vecs = oi.eig_topk(k, h=h)
    T = H @ H.conj().T
    lam = torch.linalg.eigvalsh(T).flip(0)[:k]
    top = float(lam[0])
    assert float((vals - lam.clamp(min=0)).abs().max()) < 1e-12 * top
    assert float((T @ vecs - vecs * vals).norm(dim=0).max()) < 1e-12 * top


@pytest.mark.parametrize('n', [64, 130, 961, 2400])
@pytest.mark.parametrize('live', ['one', 'few', 'most', 'ends'])
def test_dense_with_zero_rows(n, live):
    """Zero rows and columns scattered over T, as of frequencies outside every pupil (a pair's residual there is its value times its rows)."""
    from opticalimaging_b200 import imaging as oi
    rng = np.random.default_rng(n)
    on = {'one': rng.permutation(n) < 1, 'few': rng.random(n) < 0.1, 'most': rng.random(n) < 0.9,
          'ends': np.arange(n) % (n - 1) == 0}[live]
    h = (rng.standard_normal((n, 40)) + 1j * rng.standard_normal((n, 40))) * on[:, None] * 2.0 ** -np.arange(40)
    T = torch.from_numpy(h @ h.conj().T).cuda()
    vals, vecs = oi.eig_topk(4, tcc=T)
    lam = torch.from_numpy(np.linalg.svd(h, compute_uv=False)[:4] ** 2).cuda()
    top = float(lam[0])
    assert float((vals - lam).abs().max()) < 1e-12 * top
    assert float((T @ vecs - vecs * vals).norm(dim=0).max()) < 1e-12 * top


def test_small_blocks_and_the_iteration_limit():
    """The C entry with a block of fewer than 64 vectors, and a limit it cannot meet: the status says so."""
    from opticalimaging_b200 import _native as N
    n, p, k = 90, 10, 4
    g = torch.Generator().manual_seed(7)
    U = torch.linalg.qr(torch.randn((n, n), generator=g, dtype=torch.complex128))[0]
    lam = 0.5 ** torch.arange(n, dtype=torch.float64)
    T = ((U * lam) @ U.conj().T).cuda().contiguous()
    nbytes = ctypes.c_longlong(0)
    N.call('oi_eig_topk64_workspace', n, p, 0, 0, ctypes.byref(nbytes))
    work = torch.empty(nbytes.value, dtype=torch.uint8, device='cuda')
    vecs = torch.empty((n, k), dtype=torch.complex128, device='cuda')
    vals = torch.empty(k, dtype=torch.float64, device='cuda')
    iters = ctypes.c_int(0)
    for limit, met in ((300, True), (1, False)):
        N.call('oi_eig_topk64', N.ptr(T), None, 0, n, n, k, p, limit, 1e-13, N.ptr(vecs), N.ptr(vals), N.ptr(work),
               nbytes.value, ctypes.byref(iters), N.stream_handle())
        torch.cuda.synchronize()
        assert (iters.value > 0) == met and abs(iters.value) <= limit
        if met:
            assert float((vals.cpu() - lam[:k]).abs().max()) < 2e-13


def test_values_that_are_not_numbers_come_back_as_such():
    from opticalimaging_b200 import imaging as oi
    T = torch.eye(128, dtype=torch.complex128, device='cuda')
    T[100, 3] = float('nan')
    _, vecs = oi.eig_topk(4, tcc=T)
    assert bool(torch.isnan(torch.view_as_real(vecs)).any())
