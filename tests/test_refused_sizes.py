"""Sizes the native entry points refuse before any launch (on a machine without a GPU, where a launch would end in another
error)."""
import ctypes

import pytest
import torch

from opticalimaging_b200 import _native as N

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason='host pointers: an unrefused call would be launched')
EINVAL, ERANGE = -1, -3
BUFFER = ctypes.create_string_buffer(4096)


def test_complex_fields_of_more_than_65535_channels():
    p = ctypes.addressof(BUFFER)
    for batch, nch in ((65536, 1), (22000, 3)):
        rc = N.load().oi_band_spectrum_fft_c64(p, batch, 256, 256, nch, -2, 5, -2, 5, p, p, 1.0, p, p, None)
        assert rc == ERANGE


@pytest.mark.parametrize('entry', ['oi_coarse_to_image', 'oi_coarse_to_image_fft'])
def test_partial_sums_that_are_not_whole_vectors(entry):
    p = ctypes.addressof(BUFFER)
    lib = N.load()
    if entry == 'oi_coarse_to_image':
        rc = lib.oi_coarse_to_image(p, 2, 1, 3, 3, 2, 2, p, p, p, p, 9, 9, p, p, None)
    else:
        rc = lib.oi_coarse_to_image_fft(p, 2, 1, 3, 3, 2, 2, p, p, None, None, p, p, 256, 256, p, p, p, None)
    assert rc == EINVAL
