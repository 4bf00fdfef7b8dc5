"""Inverse lithography (ILT) and source-mask optimisation (SMO) around the adjoint kernel.

* ``ResistModel``: the sigmoid threshold resist R(I) = sigmoid(a (I - threshold)) of the inverse-lithography
  study (steepness a = 50, threshold 0.25).
* ``optimize_mask``: pixel-based ILT.  The mask transmission is m = sigmoid(logits); the loss is
  ||R(I(m)) - target||^2 summed over pixels and focus planes; Adam steps on the logits, the gradient through
  ``autograd.aerial_image`` (the hand-written adjoint, no stored per-field arrays).  Works with SOCS kernels and
  with Abbe models.
* ``optimize_source_mask``: source-mask co-optimisation on an Abbe model.  Source weights are v = exp(s) (kept
  positive); each iteration takes one Adam step on the mask logits and one on s, both gradients at the same
  point: the mask's through the adjoint, the source's from ``source_weight_gradient`` (dI/dv_j =
  (n I_j - I) / sum v, CalculateAerialImage.py:89-92).  A source update only rescales the model's field weights
  (``set_source_weights``, weight of point j = n v_j / sum v); the pupils stay resident.

The reference has no optimisation loop; it differentiates its SOCS image by torch autograd
(CalculateAerialImage_SOCS.py:3-11), which the adjoint reproduces (tests/test_adjoint_gpu.py).
"""
from __future__ import annotations

import ctypes
import functools

import torch
from torch.autograd import forward_ad

from . import _native as N
from .autograd import aerial_image, source_weight_gradient
from .engine import CoherentModel


class ResistModel:
    """Sigmoid threshold resist: R(I) = sigmoid(steepness (I - threshold))."""

    def __init__(self, steepness: float = 50.0, threshold: float = 0.25):
        self.steepness, self.threshold = float(steepness), float(threshold)

    def __call__(self, image: torch.Tensor) -> torch.Tensor:
        return torch.sigmoid(self.steepness * (image - self.threshold))


@functools.cache
def _loss_workspace() -> int:
    """Bytes of the loss kernel's partial sums (the library's own constant)."""
    nbytes = ctypes.c_longlong(0)
    N.call('oi_resist_loss_workspace', ctypes.byref(nbytes))
    return nbytes.value


class _ResistTerms(torch.autograd.Function):
    """(loss, D, s) in one pass over the images: loss = sum (s - target)^2, s = sigmoid(a (I - thr)), D = dloss/dI.

    With q = a s (1 - s): dloss = D dI, ds = q dI, dD = (2 q^2 + a D (1 - 2 s)) dI.  D and s are outputs, so that a
    backward pass that is itself recorded (create_graph) differentiates through them, to any order, and neither the
    image nor the target is kept: what the caller does with them afterwards changes no derivative."""

    @staticmethod
    def forward(ctx, image, target, steepness, threshold):
        img = image.contiguous()
        B, Z, ny, nx = img.shape
        grad, s = (torch.empty_like(img), torch.empty_like(img)) if ctx.needs_input_grad[0] else (None, None)
        loss = torch.empty((), dtype=torch.float32, device=img.device)
        nbytes = _loss_workspace()
        work = torch.empty(nbytes, dtype=torch.uint8, device=img.device)
        N.call('oi_resist_loss_terms', N.ptr(img), N.ptr(target), B, Z, ny * nx, steepness, threshold, N.ptr(grad), N.ptr(s),
               N.ptr(loss), N.ptr(work), nbytes, N.stream_handle(img.device))
        if grad is not None:
            ctx.set_materialize_grads(False)
            ctx.steepness = steepness
            ctx.save_for_backward(grad, s)
        return loss, grad, s

    @staticmethod
    def backward(ctx, g_loss, g_grad, g_s):
        d, s = ctx.saved_tensors
        g = None if g_loss is None else d * g_loss
        if g_grad is not None or g_s is not None:   # from a recorded backward pass
            a = ctx.steepness
            q = a * s * (1.0 - s)
            for g_out, slope in ((g_grad, 2.0 * q * q + a * d * (1.0 - 2.0 * s)), (g_s, q)):
                if g_out is not None:
                    g = g_out * slope if g is None else g + g_out * slope
        return g, None, None, None


class _ResistLoss:
    """sum (sigmoid(a (I - thr)) - target)^2 with its derivatives by the images."""

    @staticmethod
    def apply(image, target, steepness, threshold):
        return _ResistTerms.apply(image, target, steepness, threshold)[0]


def _differentiated(t: torch.Tensor) -> bool:
    """Whether autograd follows t, backward or forward (a dual tensor)."""
    return t.requires_grad or forward_ad.unpack_dual(t).tangent is not None


def ilt_loss(model: CoherentModel, mask: torch.Tensor, target: torch.Tensor, resist: ResistModel):
    """(loss, image): ||R(I(mask)) - target||^2 over pixels and planes; mask [B, ny, nx], target [B, ny, nx]."""
    image = aerial_image(model, mask)                        # [B, Z, ny, nx]
    # one float32 target per mask and the sigmoid resist itself, its parameters plain numbers: the fused loss; any other
    # resist callable, parameters that are tensors (they may want a gradient, or differ by pixel), broadcast or
    # differentiable target: torch operations
    if (type(resist) is ResistModel and isinstance(resist.steepness, (int, float))
            and isinstance(resist.threshold, (int, float)) and target.dtype == torch.float32 and target.device == image.device
            and target.shape == (image.shape[0],) + image.shape[2:] and target.is_contiguous()
            and not _differentiated(target)):
        return _ResistLoss.apply(image, target, float(resist.steepness), float(resist.threshold)), image
    loss = torch.sum((resist(image) - target[:, None]) ** 2)
    return loss, image


def _check_target(model: CoherentModel, target: torch.Tensor) -> torch.Tensor:
    if target.dim() != 3 or target.shape[1:] != (model.ny, model.nx):
        raise ValueError(f'target must be [B, {model.ny}, {model.nx}]')
    return target.to(model.device, torch.float32).contiguous()


def optimize_mask(model: CoherentModel, target: torch.Tensor, logits: torch.Tensor | None = None, steps: int = 50,
                  lr: float = 0.1, resist: ResistModel | None = None):
    """Pixel-based ILT: Adam on the mask logits for `steps` iterations.  Returns (mask, losses), mask =
    sigmoid(logits) [B, ny, nx] and the loss before each step.  Default start: logits = 4 (target - 1/2)."""
    resist = resist or ResistModel()
    target = _check_target(model, target)
    if logits is None:
        logits = 4.0 * (target - 0.5)
    logits = logits.to(model.device, torch.float32).detach().clone().requires_grad_(True)
    opt = torch.optim.Adam([logits], lr=lr)
    losses = []
    for _ in range(steps):
        opt.zero_grad()
        loss, _ = ilt_loss(model, torch.sigmoid(logits), target, resist)
        loss.backward()
        opt.step()
        losses.append(loss.item())
    return torch.sigmoid(logits).detach(), losses


def set_source_weights(model: CoherentModel, values: torch.Tensor, index_image: float) -> None:
    """Re-weight an Abbe model for source weights `values` [S] (the order of Calc_SourceSimple's Value): field
    (point j, component e) of every plane gets n v_j / sum v.  The pupils do not depend on the weights."""
    if model.kind != 'abbe':
        raise ValueError('source weights belong to an Abbe model (abbe_model)')
    Z, K = model.weights.shape
    w = model.weights
    S, P = values.numel(), getattr(model, 'pol_states', 1)      # fields are [polarisation state][point][component]
    if K % (P * S):
        raise ValueError(f'{S} source weights do not divide the model\'s {K} fields')
    v = values.to(model.device, torch.float64).reshape(-1).contiguous()
    if (w.dtype == torch.float32 and w.is_contiguous()
            and not (_differentiated(w) or _differentiated(v) or w.is_inference())):
        N.call('oi_source_weights', N.ptr(v), S, K // (P * S), K, Z, float(index_image), N.ptr(w),
               N.stream_handle(model.device))
        torch.autograd.graph.increment_version(w)   # an in-place change, to whatever has saved the weights
    else:   # what autograd has to see or to refuse
        per = ((index_image / v.sum()) * v).repeat_interleave(K // (P * S)).repeat(P)
        w.copy_(per.to(torch.float32)[None].expand(Z, K))
    model.packed = None   # packed for the previous weights


def optimize_source_mask(model: CoherentModel, values: torch.Tensor, index_image: float, target: torch.Tensor,
                         logits: torch.Tensor | None = None, steps: int = 30, lr_mask: float = 0.1,
                         lr_source: float = 0.05, resist: ResistModel | None = None):
    """SMO on an Abbe model: per iteration one Adam step on the mask logits and one on the source log-weights,
    both gradients taken at the same point.  Returns (mask, source weights [S], losses).  The model's weights are
    left set to the returned source."""
    if model.kind != 'abbe':
        raise ValueError('source-mask optimisation needs an Abbe model (abbe_model)')
    resist = resist or ResistModel()
    target = _check_target(model, target)
    if logits is None:
        logits = 4.0 * (target - 0.5)
    logits = logits.to(model.device, torch.float32).detach().clone().requires_grad_(True)
    s = torch.log(values.to(model.device, torch.float64).reshape(-1).clamp_min(1e-12)).requires_grad_(True)
    opt_m = torch.optim.Adam([logits], lr=lr_mask)
    opt_s = torch.optim.Adam([s], lr=lr_source)
    losses = []
    for _ in range(steps):
        v = torch.exp(s.detach())
        set_source_weights(model, v, index_image)
        opt_m.zero_grad()
        opt_s.zero_grad()
        mask = torch.sigmoid(logits)
        loss, image = ilt_loss(model, mask, target, resist)
        image.retain_grad()
        loss.backward()                                       # dL/dlogits and dL/dI
        gv = source_weight_gradient(model, mask.detach(), image.grad, v, index_image)   # [B, S]
        s.grad = gv.sum(dim=0).to(torch.float64) * v          # dL/ds = dL/dv * v
        opt_m.step()
        opt_s.step()
        losses.append(loss.item())
    v = torch.exp(s.detach())
    set_source_weights(model, v, index_image)
    return torch.sigmoid(logits).detach(), v.float(), losses
