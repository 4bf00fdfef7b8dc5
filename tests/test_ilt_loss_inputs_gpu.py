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


def test_source_gradient_with_a_tangent():
    from opticalimaging_b200.engine import Band, CoherentModel
    from opticalimaging_b200.autograd import source_weight_gradient
    g = torch.Generator(device='cuda').manual_seed(2)
    S, n = 5, 256
    pupils = torch.randn((1, S, 9, 9), generator=g, dtype=torch.complex64, device='cuda')
    model = CoherentModel(pupils, torch.ones((1, S), device='cuda'), Band(-4, 9, -4, 9), n, n, 'abbe')
    mask, grad = torch.rand((2, n, n), generator=g, device='cuda'), torch.randn((2, 1, n, n), generator=g, device='cuda')
    v = 0.5 + torch.rand(S, generator=g, dtype=torch.float64, device='cuda')
    t = torch.randn(S, generator=g, dtype=torch.float64, device='cuda')
    at = lambda v: source_weight_gradient(model, mask, grad, v, 1.3)  # noqa: E731
    with fwd.dual_level():
        value, tangent = fwd.unpack_dual(at(fwd.make_dual(v, t)))
    step = 1e-3
    want = (at(v + step * t).double() - at(v - step * t).double()) / (2 * step)
    # the central difference: FP32 results 2e-3 apart, and its own error of step^2
    top = float(value.abs().max())
    assert float((value - at(v)).abs().max()) < 1e-6 * top
    assert tangent is not None and float((tangent - want).abs().max()) < 1e-3 * top
