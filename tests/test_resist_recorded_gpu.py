"""The resist loss where the caller goes on with its tensors: changed in place before a recorded backward pass, released,
or differentiated in a batch."""
import gc
import weakref

import pytest
import torch

pytestmark = pytest.mark.gpu


def _loss(image, target, a, thr):
    return torch.sum((torch.sigmoid(a * (image - thr)) - target[:, None]) ** 2)


def _inputs():
    g = torch.Generator(device='cuda').manual_seed(3)
    leaf = torch.rand((2, 2, 8, 9), generator=g, device='cuda', requires_grad=True)
    target = (torch.rand((2, 8, 9), generator=g, device='cuda') > 0.5).float()
    return leaf, target, torch.randn(leaf.shape, generator=g, device='cuda')


def _derivatives(loss, leaf, v):
    """The gradient, recorded, and those of its products with v, to the third order."""
    out = [torch.autograd.grad(loss, leaf, create_graph=True)[0]]
    for _ in range(2):
        out.append(torch.autograd.grad((out[-1] * v).sum(), leaf, create_graph=True)[0])
    return [x.detach() for x in out]


@pytest.mark.parametrize('change', ['none', 'target', 'image', 'both'])
def test_recorded_backward_after_a_change_in_place(change):
    from opticalimaging_b200.ilt import _ResistLoss
    leaf, target, v = _inputs()
    a = 8.0
    want = _derivatives(_loss(leaf.double(), target.double(), a, 0.3), leaf, v)
    image = leaf * 1.0
    loss = _ResistLoss.apply(image, target, a, 0.3)
    with torch.no_grad():
        if change in ('target', 'both'):
            target.zero_()
        if change in ('image', 'both'):
            image.mul_(-2.0)
    got = _derivatives(loss, leaf, v)
    # a |I - thr| <= 5.6: each derivative is a sum of a few FP32 products of s to 2^-24 relative with factors a^order
    for order, (x, y) in enumerate(zip(got, want), 1):
        assert float((x - y).abs().max()) < 2e-6 * a ** order * 5


def test_keeps_nothing_of_the_callers():
    from opticalimaging_b200.ilt import _ResistLoss
    leaf, target, _ = _inputs()
    image = leaf * 1.0
    loss = _ResistLoss.apply(image, target, 8.0, 0.3)
    refs = [weakref.ref(image), weakref.ref(target)]
    del image, target
    gc.collect()
    assert loss.requires_grad and all(r() is None for r in refs)


def test_batched_backward():
    from opticalimaging_b200.ilt import _ResistLoss
    leaf, target, _ = _inputs()
    loss = _ResistLoss.apply(leaf, target, 8.0, 0.3)
    one, = torch.autograd.grad(loss, leaf, retain_graph=True)
    many, = torch.autograd.grad(loss, leaf, grad_outputs=torch.tensor([1.0, -2.0], device='cuda'), is_grads_batched=True)
    assert torch.equal(many[0], one) and torch.equal(many[1], -2.0 * one)
