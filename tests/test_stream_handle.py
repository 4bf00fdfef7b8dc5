"""Native calls take the stream of a CUDA device only: with host tensors they end in an error before the library is called
(no GPU needed: the device queries are faked)."""
import pytest
import torch

from opticalimaging_b200 import _native as N
from opticalimaging_b200 import engine, imaging
from opticalimaging_b200.params import Numerics


@pytest.fixture
def calls(monkeypatch):
    made = []
    monkeypatch.setattr(torch.cuda, 'current_device', lambda: 1)
    monkeypatch.setattr(torch._C, '_cuda_getCurrentRawStream', lambda i: 100 + i, raising=False)
    real = N.call
    monkeypatch.setattr(N, 'call', lambda name, *a: real(name, *a) if name.endswith('_workspace') else made.append(name))
    return made


def test_handles():
    with pytest.raises(ValueError):
        N.stream_handle(torch.device('cpu'))
    with pytest.raises(ValueError):
        N.stream_handle('cpu')


def test_cuda_devices(calls):
    assert N.stream_handle() == 101 and N.stream_handle('cuda') == 101 and N.stream_handle(torch.device('cuda', 3)) == 103


@pytest.mark.parametrize('use', [
    lambda: engine.twiddle(4, 4, 0, 0, 4, 1, 'cpu'),
    lambda: imaging.eig_topk(2, tcc=torch.eye(80, dtype=torch.complex128)),
    lambda: imaging.eig_topk(2, h=torch.ones((1, 80, 9), dtype=torch.complex128)),
    lambda: imaging.socs_kernels_from_pupils(torch.ones((1, 25, 30), dtype=torch.complex128), [5, 5], [64, 64], Numerics())])
def test_host_tensors_do_not_reach_the_library(calls, use):
    with pytest.raises(ValueError):
        use()
    assert not calls
