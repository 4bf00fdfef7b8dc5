"""mask_gradient_from_w hands the native code a contiguous complex64 array [B, br, bc] of the model's band, whatever it is
given: other types are converted, conjugate views resolved, values broadcast as an assignment to the band does, and any
other shape is refused before the native code sees it."""
import ctypes
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from opticalimaging_b200 import autograd as A
from opticalimaging_b200.engine import Band

BAND = Band(-2, 5, -1, 4)
SHAPE = (3, BAND.br, BAND.bc)


@pytest.fixture
def handed(monkeypatch):
    """The arrays handed to oi_hermitian_half (on the CPU, in its place)."""
    seen = []

    def call(name, w, n, batch, nz, m0r, br, m0c, bc, scale, half, stream):
        assert name == 'oi_hermitian_half' and (n, nz) == (1, 1)
        raw = (ctypes.c_float * (2 * batch * br * bc)).from_address(w)
        seen.append(np.array(raw, dtype=np.float32).view(np.complex64).reshape(batch, br, bc))

    monkeypatch.setattr(A, 'N', SimpleNamespace(call=call, ptr=lambda t: t.data_ptr(), stream_handle=lambda d=None: 0))
    monkeypatch.setattr(A, '_half_spectrum_to_image', lambda half, *a: half)
    return seen


def _model():
    return SimpleNamespace(band=BAND, ny=16, nx=16, device=torch.device('cpu'))


def _w(shape, dtype=torch.complex64):
    g = torch.Generator().manual_seed(1)
    return torch.randn(shape, generator=g, dtype=torch.complex128).to(dtype)


@pytest.mark.parametrize('make', [
    lambda: _w(SHAPE), lambda: _w(SHAPE, torch.complex128), lambda: _w(SHAPE).conj(), lambda: _w(SHAPE).real.double(),
    lambda: _w((3, 4, 5)).transpose(1, 2), lambda: _w((3, 1, 4)), lambda: _w((3, 1, 1)).conj()])
def test_arrays_of_the_band(handed, make):
    w = make()
    A.mask_gradient_from_w(_model(), w)
    want = np.broadcast_to(w.resolve_conj().numpy(), SHAPE).astype(np.complex64)
    assert len(handed) == 1 and np.array_equal(handed[0], want)


@pytest.mark.parametrize('shape', [(3, 4, 4), (3, 5, 3), (3, 6, 4), (2, 3, 5, 4), (20,)])
def test_other_shapes_are_refused(handed, shape):
    with pytest.raises((RuntimeError, ValueError)):
        A.mask_gradient_from_w(_model(), _w(shape))
    assert not handed
