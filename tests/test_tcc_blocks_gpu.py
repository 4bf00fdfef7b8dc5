"""TCC assembly that skips the zero blocks of the pupil matrix, against torch in FP64: sizes around the 64-row tiles and
the 16-point chunks, supports that leave whole blocks empty, and values that are not finite beside zero blocks."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _assemble(h, marked):
    from opticalimaging_b200 import _native as N
    ne, n, s = h.shape
    out = torch.full((n, n), 7.0, dtype=torch.complex128, device='cuda')
    if marked:
        nbytes = ctypes.c_longlong(0)
        N.call('oi_tcc_assemble64_marked_workspace', ne, n, s, ctypes.byref(nbytes))
        work = torch.full((nbytes.value,), 255, dtype=torch.uint8, device='cuda')
        N.call('oi_tcc_assemble64_marked', N.ptr(h), ne, n, s, N.ptr(out), N.ptr(work), nbytes.value, N.stream_handle())
    else:
        N.call('oi_tcc_assemble64', N.ptr(h), ne, n, s, N.ptr(out), N.stream_handle())
    return out


def _window(ne, n, s, width):
    rng = np.random.default_rng(n + s)
    h = rng.standard_normal((ne, n, s)) + 1j * rng.standard_normal((ne, n, s))
    row, col = np.arange(n)[:, None] / n, np.arange(s)[None, :] / max(s, 2)
    return torch.from_numpy(h * (np.abs(row - 0.2 - 0.6 * col) < width)).cuda()


@pytest.mark.parametrize('ne', [1, 3])
@pytest.mark.parametrize('n,s', [(1, 1), (15, 16), (64, 17), (65, 33), (200, 100), (961, 520)])
@pytest.mark.parametrize('width', [0.02, 0.25, 2.0])
@pytest.mark.parametrize('marked', [True, False])
def test_matches_fp64_product(ne, n, s, width, marked):
    h = _window(ne, n, s, width)
    got = _assemble(h, marked)
    want = sum(e @ e.conj().T for e in h)
    # sums of ne * s products of O(1) values, each rounded to 2^-53
    assert float((got - want).abs().max()) <= 1e-15 * (ne * s) * float(h.abs().max()) ** 2
    assert torch.equal(got, got.conj().T.contiguous()) or bool((got.diagonal().imag.abs() < 1e-12).all())


def test_values_that_are_not_finite_reach_every_product():
    """0 times NaN counts: the marked form leaves out only blocks whose other side is finite."""
    h = _window(1, 200, 100, 0.1)
    h[0, 150, 90] = float('nan')
    a, b = _assemble(h, True), _assemble(h, False)
    assert torch.equal(torch.isnan(a.real), torch.isnan(b.real)) and bool(torch.isnan(a.real).any())
