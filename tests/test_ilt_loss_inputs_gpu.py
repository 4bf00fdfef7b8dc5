"""ilt_loss with a resist whose parameters are tensors, and with a target that carries a tangent."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from tests.fixtures import load

pytestmark = pytest.mark.gpu


def _setup():
    from opticalimaging_b200.engine import SocsKernels
    meta, a = load('autograd')
    model = SocsKernels.from_full_grid(torch.from_numpy(a['kernels']).cuda())
    mask = torch.sigmoid(torch.from_numpy(a['logits']).cuda())[None].float()
    return model, mask, torch.from_numpy(a['target']).cuda().float()[None]


@pytest.mark.parametrize('name', ['threshold', 'steepness'])
@pytest.mark.parametrize('per_pixel', [False, True])
def test_resist_parameters_that_are_tensors(name, per_pixel):
    from opticalimaging_b200 import ilt
    model, mask, target = _setup()
    resist = ilt.ResistModel(30.0, 0.25)
    shape = target.shape[1:] if per_pixel else ()
    value = torch.full(shape, getattr(resist, name), device='cuda', requires_grad=True)
    setattr(resist, name, value)
    loss, image = ilt.ilt_loss(model, mask, target, resist)
    loss.backward()
    v64 = value.detach().double().requires_grad_(True)
    a, thr = (v64, 0.25) if name == 'steepness' else (30.0, v64)
    l64 = torch.sum((torch.sigmoid(a * (image.detach().double() - thr)) - target.double()[:, None]) ** 2)
    l64.backward()
    # FP32 sums of up to ny * nx terms of one order of magnitude
    assert value.grad is not None and abs(float(loss) - float(l64)) < 1e-5 * float(l64)
    assert float((value.grad - v64.grad).abs().max()) < 1e-4 * float(v64.grad.abs().max())


def test_target_with_a_tangent():
    from opticalimaging_b200 import ilt
    model, mask, target = _setup()
    with fwd.dual_level():
        v = torch.randn(target.shape, generator=torch.Generator(device='cuda').manual_seed(1), device='cuda')
        loss, image = ilt.ilt_loss(model, mask, fwd.make_dual(target, v), ilt.ResistModel(30.0, 0.25))
        got = fwd.unpack_dual(loss).tangent
    r = torch.sigmoid(30.0 * (image.double() - 0.25)) - target.double()[:, None]
    want = float((-2.0 * r * v[:, None]).sum())
    # an FP32 sum of ny * nx terms of both signs
    assert got is not None and abs(float(got) - want) < 1e-5 * float((2.0 * r * v[:, None]).abs().sum())
