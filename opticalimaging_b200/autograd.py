"""Differentiable aerial images for inverse lithography.

``aerial_image(model, mask)`` is the batched image of a resident ``CoherentModel`` (SOCS kernels or Abbe
pupils) as a ``torch.autograd.Function``: its backward runs the hand-written adjoint (``oi_coherent_adjoint``),
so a loss on the image -- e.g. a sigmoid resist model against a target -- differentiates into the mask
transmission without storing any per-field array (the forward is recomputed inside the adjoint).

``source_weight_gradient(...)`` gives dL/dv_j for the source-point weights v_j of an Abbe model through the
linear Abbe identity dI/dv_j = (n I_j - I) / sum(v) (CalculateAerialImage.py:89-92): the gradient of the
untruncated image.  For a SOCS model the truncated kernels depend on the source through the eigenvectors,
so its source gradient is taken as that of the untruncated (Abbe) image, which is what it approximates.

The reference obtains gradients by torch autograd through its FFTs (CalculateAerialImage_SOCS.py:3-11); the
tests compare both, and central finite differences in FP64.
"""
from __future__ import annotations

import torch
from torch.autograd import forward_ad

from . import _native as N
from .engine import Band, CoherentModel, Plan, band_spectrum, coherent_image, field_split_sm


def _half_spectrum_to_image(ihat: torch.Tensor, br: int, bc: int, ny: int, nx: int) -> torch.Tensor:
    """Real images [count, ny, nx] from Hermitian halves ihat [count, 2br-1, bc] (qc > 0 already doubled)."""
    dev = ihat.device
    count = ihat.shape[0]
    plan = Plan.get(ny, nx, Band(-(br - 1), br, 0, bc), dev)
    out = torch.empty((count, ny, nx), dtype=torch.float32, device=dev)
    ih = ihat.contiguous()
    s = N.stream_handle(dev)
    if plan.fft:
        v = torch.empty(count * bc * ny, dtype=torch.complex64, device=dev)
        N.call('oi_spectrum_to_image_fft', N.ptr(ih), count, br, bc, N.ptr(plan.wn_y), N.ptr(plan.wn_x), ny, nx,
               N.ptr(v), N.ptr(out), s)
    else:
        N.call('oi_spectrum_to_image', N.ptr(ih), count, br, bc, N.ptr(plan.sy), N.ptr(plan.sx), ny, nx, N.ptr(out), s)
    return out


ADJOINT_COARSE = (128, 128)


def adjoint_plan(model: CoherentModel) -> Plan:
    """The model's plan on the 128 x 128 coarse grid the adjoint kernel works on (exact for bands up to 64)."""
    b = model.band
    if 2 * b.br - 1 > ADJOINT_COARSE[0] or 2 * b.bc - 1 > ADJOINT_COARSE[1]:
        raise NotImplementedError(f'the adjoint covers bands up to 64 x 64 (this one is {b.br} x {b.bc})')
    return Plan.get(model.ny, model.nx, b, model.device, coarse=ADJOINT_COARSE)


def coarse_gradient(model: CoherentModel, g: torch.Tensor) -> torch.Tensor:
    """The band-limited coarse copy g^c [B, Z, Mr, Mc] of g = dL/dI [B, Z, ny, nx]:
    g^c(s) = 1/(Mr Mc) sum_{|qr|<br, |qc|<bc} ghat(q) exp(-2 pi i q.s/M), ghat(q) = sum_r g(r) exp(+2 pi i q.r/N)."""
    plan = adjoint_plan(model)
    return _coarse_gradient(model, g, 1.0 / (plan.mr * plan.mc))


def _coarse_gradient(model: CoherentModel, g: torch.Tensor, scale: float) -> torch.Tensor:
    """scale * sum_q ghat(q) exp(-2 pi i q.s/M) on the adjoint's coarse grid."""
    b, plan = model.band, adjoint_plan(model)
    B, Z = g.shape[0], g.shape[1]
    ny, nx = model.ny, model.nx
    ib = Band(-(b.br - 1), 2 * b.br - 1, 0, b.bc)                     # image band, Hermitian half in x
    gplan = Plan.get(ny, nx, ib, model.device)
    g = g.reshape(B * Z, ny, nx).contiguous()
    if gplan.fft:
        t = torch.empty(B * Z * b.bc * (ny + plan.mr), dtype=torch.complex64, device=model.device)
        gc = torch.empty((B, Z, plan.mr, plan.mc), dtype=torch.float32, device=model.device)
        N.call('oi_coarse_gradient_fft', N.ptr(g), B * Z, ny, nx, b.br, b.bc, N.ptr(gplan.wn_x), N.ptr(gplan.wn_y),
               N.ptr(plan.coarse_fft_tables()[0]), N.ptr(plan.wm_c), scale, N.ptr(t), N.ptr(gc), N.stream_handle(model.device))
        return gc
    gh = band_spectrum(g, N.FIELD_REAL_F32, gplan, scale=scale * ny * nx)[:, 0]   # [B*Z, 2br-1, bc]
    gh[:, :, 1:] *= 2.0
    return _half_spectrum_to_image(gh, b.br, b.bc, plan.mr, plan.mc).view(B, Z, plan.mr, plan.mc)


def _adjoint_shares(model: CoherentModel, band: torch.Tensor, gc: torch.Tensor, pupils, weights):
    """W in shares [nsplit, B, Z, nch, br, bc] over the fields `pupils` [Z, K, br, bc] weighted by `weights`."""
    b, plan = model.band, adjoint_plan(model)
    B, nch = band.shape[0], band.shape[1]
    Z, K = pupils.shape[0], pupils.shape[1]
    nsplit = field_split_sm(K * nch, B * Z)
    wout = torch.empty((nsplit, B, Z, nch, b.br, b.bc), dtype=torch.complex64, device=model.device)
    N.call('oi_coherent_adjoint', N.ptr(band), B, nch, b.m0r, b.br, b.m0c, b.bc, N.ptr(pupils), N.ptr(weights), Z, K,
           N.ptr(gc), plan.mr, plan.mc, N.ptr(plan.wm_r), N.ptr(plan.wm_c), nsplit, N.ptr(wout), None,
           N.stream_handle(model.device))
    return wout


def _field_dots(model: CoherentModel, band: torch.Tensor, gc: torch.Tensor) -> torch.Tensor:
    """<g, |E_f|^2> of every field f of the model: [B, Z, K*nch]."""
    b, plan = model.band, adjoint_plan(model)
    B, nch = band.shape[0], band.shape[1]
    Z, K = model.planes, model.count
    nsplit = field_split_sm(K * nch, B * Z)
    gc = gc.contiguous()
    dots = torch.empty((B, Z, K * nch), dtype=torch.float32, device=model.device)
    N.call('oi_coherent_field_dots', N.ptr(band), B, nch, b.m0r, b.br, b.m0c, b.bc, N.ptr(model.pupils),
           N.ptr(model.weights), Z, K, N.ptr(gc), plan.mr, plan.mc, N.ptr(plan.wm_r), N.ptr(plan.wm_c), nsplit, N.ptr(dots),
           N.stream_handle(model.device))
    return dots


def coherent_adjoint(model: CoherentModel, band: torch.Tensor, gc: torch.Tensor, field_dots: bool = False):
    """W [B, nch, br, bc] (summed over planes) and, optionally, field dots [B, Z, K*nch]."""
    gc = gc.contiguous()
    w = _adjoint_shares(model, band, gc, model.pupils, model.weights).sum(dim=(0, 2))
    return w, (_field_dots(model, band, gc) if field_dots else None)


def mask_gradient_from_w(model: CoherentModel, w: torch.Tensor) -> torch.Tensor:
    """dL/dt [B, ny, nx] = 2/(ny nx) Re sum_{m in band} W(m) exp(-2 pi i m.y/N) for W [B, br, bc] (of any type and device;
    [B, 1, bc] and the like are broadcast)."""
    full = torch.empty((w.shape[0], model.band.br, model.band.bc), dtype=torch.complex64, device=model.device).copy_(w)
    return _mask_gradient(model, full[None, :, None], 2.0 / (model.ny * model.nx))


def _mask_gradient(model: CoherentModel, shares: torch.Tensor, scale: float) -> torch.Tensor:
    """scale Re sum_m W(m) exp(-2 pi i m.y/N) [B, ny, nx], W the sum of shares [n, B, Z, br, bc] over n and Z."""
    b = model.band
    n, B, Z = shares.shape[0], shares.shape[1], shares.shape[2]
    R = max(abs(b.m0r), abs(b.m0r + b.br - 1))
    C = max(abs(b.m0c), abs(b.m0c + b.bc - 1))
    half = torch.empty((B, 2 * R + 1, C + 1), dtype=torch.complex64, device=shares.device)
    N.call('oi_hermitian_half', N.ptr(shares), n, B, Z, b.m0r, b.br, b.m0c, b.bc, float(scale), N.ptr(half),
           N.stream_handle(model.device))
    return _half_spectrum_to_image(half, R + 1, C + 1, model.ny, model.nx)


class _CoherentImage(torch.autograd.Function):
    @staticmethod
    def forward(ctx, mask, model):
        ctx.model = model
        with torch.no_grad():
            m = mask.detach().contiguous()
            model.check_grid(m)
            band = band_spectrum(m, N.FIELD_REAL_F32, model.plan, form=model.form)
            image = coherent_image(band, *model.fields_for(N.FIELD_REAL_F32), model.plan, form=model.form)
        # the backward pass starts from the plan's default FP32 band spectrum: the forward's own, or, for a model in another
        # form ('dft', 'bf16x3'), one of its own
        ctx.save_for_backward(mask, band if model.form in (None, 'fft') else None)
        return image                                                        # [B, Z, ny, nx] for every model

    @staticmethod
    def backward(ctx, g):
        mask, band = ctx.saved_tensors
        model = ctx.model
        with torch.no_grad():
            if band is None:
                band = band_spectrum(mask.detach().contiguous(), N.FIELD_REAL_F32, model.plan)
            # g^c without its 1 / (ny nx) -> the factor (ny nx) / (Mr Mc) moves to the last scale; a real mask's
            # gradient is the same through the packed fields, which give the same image for every real mask
            plan = adjoint_plan(model)
            gc = _coarse_gradient(model, g.to(torch.float32), 1.0 / (model.ny * model.nx))
            w = _adjoint_shares(model, band, gc, *model.fields_for(N.FIELD_REAL_F32))
            grad = _mask_gradient(model, w[:, :, :, 0], 2.0 / (plan.mr * plan.mc))
        return grad.view_as(mask), None


def aerial_image(model: CoherentModel, mask: torch.Tensor) -> torch.Tensor:
    """Differentiable image [B, Z, ny, nx] of real float32 masks [B, ny, nx] (gradient via the adjoint kernel)."""
    if mask.dtype != torch.float32 or mask.dim() != 3:
        raise ValueError('mask must be a float32 [B, ny, nx] tensor')
    return _CoherentImage.apply(mask, model)


def source_weight_gradient(model: CoherentModel, mask: torch.Tensor, g: torch.Tensor, values: torch.Tensor,
                           index_image: float) -> torch.Tensor:
    """dL/dv [B, S] for the source weights v (the Value of Calc_SourceSimple, length S) of an Abbe model
    built from them: dI/dv_j = (n I_j - I) / sum(v), I_j = sum_e |E_{j,e}|^2 (CalculateAerialImage.py:89-92)."""
    if model.kind != 'abbe':
        raise ValueError('source_weight_gradient needs an Abbe model (abbe_model)')
    with torch.no_grad():
        band = band_spectrum(mask.contiguous(), N.FIELD_REAL_F32, model.plan)
        gc = coarse_gradient(model, g.to(torch.float32).contiguous())
        dots = _field_dots(model, band, gc)                             # [B, Z, P*S*E]
        B, Z, K = dots.shape
        S = values.numel()
        P = getattr(model, 'pol_states', 1)                              # incoherent polarisation states
        E = K // (S * P)
        if S * P * E != K:
            raise ValueError(f'{S} source weights do not divide the model\'s {K} fields')
        v = values.to(dots.device, torch.float64).reshape(-1)
        if forward_ad.unpack_dual(v).tangent is not None:   # torch operations carry the tangent
            d = dots.view(B, Z, P, S, E).sum(dim=(1, 2, 4)).double()    # <g, I_j>
            W = v.sum()
            return ((index_image * d - (d * v).sum(dim=1, keepdim=True) * index_image / W) / W).float()
        v = v.contiguous()
        out = torch.empty((B, S), dtype=torch.float32, device=dots.device)
        N.call('oi_source_gradient', N.ptr(dots), B, Z, P, S, E, N.ptr(v), float(index_image), N.ptr(out),
               N.stream_handle(dots.device))
        return out
