"""The fused resist loss, field weights and source gradient against torch in FP64: sizes off the vector width and off a
block, several planes, saturated and non-finite intensities, what the backward pass keeps, and the calls that stay with
torch operations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _loss(image, target, a, thr):
    return torch.sum((torch.sigmoid(a * (image - thr)) - target[:, None]) ** 2)


@pytest.mark.parametrize('B,Z,ny,nx', [(1, 1, 1, 1), (1, 1, 3, 5), (2, 3, 17, 23), (3, 1, 64, 64), (2, 2, 250, 301), (1, 1, 1024, 2048)])
def test_resist_loss_and_gradient(B, Z, ny, nx):
    from opticalimaging_b200.ilt import _ResistLoss
    g = torch.Generator(device='cuda').manual_seed(ny * nx)
    image = torch.rand((B, Z, ny, nx), generator=g, device='cuda')
    image[0, 0, 0, 0] = 40.0                          # saturated: exp(-a I) underflows
    target = (torch.rand((B, ny, nx), generator=g, device='cuda') > 0.5).float()
    image.requires_grad_(True)
    loss = _ResistLoss.apply(image, target, 30.0, 0.25)
    (3.0 * loss).backward()
    i64 = image.detach().double().requires_grad_(True)
    l64 = _loss(i64, target.double(), 30.0, 0.25)
    (3.0 * l64).backward()
    assert abs(float(loss) - float(l64)) < 1e-6 * float(l64) + 1e-12
    # a (I - thr) is rounded to 2^-24 of up to 30 before the exponential: 2e-6 relative of a derivative of up to 3 a / 4 * 2
    assert float((image.grad - i64.grad).abs().max()) < 3e-6 * 45


def test_resist_loss_passes_nan_and_infinity():
    from opticalimaging_b200.ilt import _ResistLoss
    image = torch.tensor([float('inf'), float('-inf'), 0.5, 0.1], device='cuda').reshape(1, 1, 2, 2).requires_grad_(True)
    target = torch.zeros((1, 2, 2), device='cuda')
    loss = _ResistLoss.apply(image, target, 30.0, 0.25)
    loss.backward()
    want = _loss(image.detach().double(), target.double(), 30.0, 0.25)
    assert abs(float(loss) - float(want)) < 1e-6 and bool((image.grad.reshape(-1)[:2] == 0).all())
    bad = torch.full((1, 1, 2, 2), float('nan'), device='cuda')
    assert bool(torch.isnan(_ResistLoss.apply(bad, target, 30.0, 0.25)))


def test_backward_kinds():
    """In-place changes after the loss, a second backward pass of a kept graph, and a recorded backward pass."""
    from opticalimaging_b200.ilt import _ResistLoss
    leaf = torch.rand((1, 2, 8, 8), device='cuda', requires_grad=True)
    target = torch.ones((1, 8, 8), device='cuda')
    image = leaf * 1.0
    loss = _ResistLoss.apply(image, target, 20.0, 0.3)
    want, = torch.autograd.grad(_loss(leaf, target, 20.0, 0.3), leaf)
    target.zero_()
    got, = torch.autograd.grad(loss, leaf, retain_graph=True)
    again, = torch.autograd.grad(loss, leaf)
    assert torch.equal(got, again) and float((got - want).abs().max()) < 1e-5
    target.fill_(1.0)
    loss = _ResistLoss.apply(leaf * 1.0, target, 20.0, 0.3)
    g, = torch.autograd.grad(loss, leaf, create_graph=True)
    h, = torch.autograd.grad(g.sum(), leaf)
    g2, = torch.autograd.grad(_loss(leaf, target, 20.0, 0.3), leaf, create_graph=True)
    h2, = torch.autograd.grad(g2.sum(), leaf)
    assert float((g - g2).abs().max()) < 1e-5 and float((h - h2).abs().max()) < 1e-3


@pytest.mark.parametrize('S,E,P,Z,B', [(1, 1, 1, 1, 1), (7, 3, 1, 2, 2), (600, 3, 2, 1, 3), (144, 1, 1, 5, 1)])
def test_source_kernels(S, E, P, Z, B):
    from opticalimaging_b200 import _native as N
    g = torch.Generator().manual_seed(S)
    v = (0.1 + torch.rand(S, generator=g, dtype=torch.float64)).cuda()
    K = P * S * E
    w = torch.empty((Z, K), device='cuda')
    N.call('oi_source_weights', N.ptr(v), S, E, K, Z, 1.3, N.ptr(w), N.stream_handle())
    per = (1.3 / v.sum() * v).repeat_interleave(E).repeat(P).float()
    assert float((w - per[None]).abs().max()) <= 2 ** -24 * float(per.max())
    dots = torch.randn((B, Z, K), generator=g).cuda()
    out = torch.empty((B, S), device='cuda')
    N.call('oi_source_gradient', N.ptr(dots), B, Z, P, S, E, N.ptr(v), 1.3, N.ptr(out), N.stream_handle())
    d = dots.double().view(B, Z, P, S, E).sum(dim=(1, 2, 4))
    want = (1.3 * d - (d * v).sum(dim=1, keepdim=True) * 1.3 / v.sum()) / v.sum()
    assert float((out - want).abs().max()) <= 1e-6 * float(want.abs().max()) + 1e-12
