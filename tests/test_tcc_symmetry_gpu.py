"""The assembled TCC is Hermitian: tiles off the diagonal are written twice from one value, exact conjugates of each other;
tiles on it to the rounding of their products."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,s', [(65, 33), (200, 100), (961, 520)])
@pytest.mark.parametrize('marked', [True, False])
def test_hermitian(n, s, marked):
    from opticalimaging_b200 import _native as N
    rng = np.random.default_rng(n)
    h = torch.from_numpy(rng.standard_normal((3, n, s)) + 1j * rng.standard_normal((3, n, s))).cuda()
    tcc = torch.full((n, n), 7.0, dtype=torch.complex128, device='cuda')
    if marked:
        nbytes = ctypes.c_longlong(0)
        N.call('oi_tcc_assemble64_marked_workspace', 3, n, s, ctypes.byref(nbytes))
        work = torch.empty(nbytes.value, dtype=torch.uint8, device='cuda')
        N.call('oi_tcc_assemble64_marked', N.ptr(h), 3, n, s, N.ptr(tcc), N.ptr(work), nbytes.value, N.stream_handle())
    else:
        N.call('oi_tcc_assemble64', N.ptr(h), 3, n, s, N.ptr(tcc), N.stream_handle())
    gap = (tcc - tcc.conj().T).abs()
    tile = torch.arange(n, device='cuda') // 64
    off = tile[:, None] != tile[None, :]
    assert float(gap[off].max()) == 0.0
    # 3 s products of O(1) values, each rounded to 2^-53, in either order
    assert float(gap[~off].max()) <= 2e-15 * 3 * s * float(h.abs().max()) ** 2
