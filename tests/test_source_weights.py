"""set_source_weights writes the model's weights as an in-place torch copy does: seen by autograd's version check, and with
the gradient or the tangent of values that have one."""
from types import SimpleNamespace

import pytest
import torch
import torch.autograd.forward_ad as fwd

from opticalimaging_b200 import ilt


def _model(device, points=4, per=3, planes=2, **kw):
    w = torch.rand((planes, points * per), device=device)
    return SimpleNamespace(kind='abbe', weights=w, device=torch.device(device), packed=(), **kw)


def _want(v, per, planes, n):
    return (n / v.sum() * v).repeat_interleave(per).float().expand(planes, -1)


def test_values_with_a_gradient():
    model = _model('cpu')
    v = torch.tensor([0.5, 1.0, 2.0, 0.25], dtype=torch.float64, requires_grad=True)
    ilt.set_source_weights(model, v, 1.3)
    x = torch.rand(model.weights.shape)
    (model.weights * x).sum().backward()
    u = v.detach().requires_grad_(True)
    (_want(u, 3, 2, 1.3) * x).sum().backward()
    assert torch.allclose(model.weights.detach(), _want(u, 3, 2, 1.3).detach()) and torch.allclose(v.grad, u.grad)
    assert model.packed is None


def test_weights_that_are_a_leaf_with_a_gradient_are_refused():
    model = _model('cpu')
    model.weights.requires_grad_(True)
    with pytest.raises(RuntimeError):
        ilt.set_source_weights(model, torch.ones(4, dtype=torch.float64), 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize('strided', [False, True])
def test_autograd_sees_the_change(strided):
    model = _model('cuda')
    if strided:
        model.weights = torch.rand((12, 2), device='cuda').t()
    v = torch.tensor([0.5, 1.0, 2.0, 0.25], dtype=torch.float64, device='cuda')
    x = torch.rand(model.weights.shape, device='cuda', requires_grad=True)
    loss = (model.weights * x).sum()
    ilt.set_source_weights(model, v, 1.3)
    assert torch.allclose(model.weights, _want(v, 3, 2, 1.3))
    with pytest.raises(RuntimeError, match='modified by an inplace operation'):
        loss.backward()


def test_values_with_a_tangent():
    model = _model('cpu')
    v = torch.tensor([0.5, 1.0, 2.0, 0.25], dtype=torch.float64)
    d = torch.tensor([1.0, -2.0, 0.5, 3.0], dtype=torch.float64)
    with fwd.dual_level():
        ilt.set_source_weights(model, fwd.make_dual(v, d), 1.3)
        w, t = fwd.unpack_dual(model.weights)
    u, j = _want(v, 3, 2, 1.3), 1.3 * (d / v.sum() - v * d.sum() / v.sum() ** 2)
    assert torch.allclose(w, u) and torch.allclose(t, j.repeat_interleave(3).float().expand(2, -1))
