"""The splat's direct caller: photon differentials on the receiver -> splat inputs -> image.

Mirror of ``model/caustics.py:224-239`` (``change_of_basis_matrix``, ``splat_photons``) on
plain ``[3, N]`` tensors:

    Mp     = 2 / (Du . (Dv x n)) * [Dv x n ; n x Du]        (2 x 3 x N)
    radius = 0.5 * max(|Du|, |Dv|)
    Ep     = 4 * flux / |Du x Dv|

so that ``Mp @ Du = (2, 0)`` and ``Mp @ Dv = (0, 2)``: the splat support is the ellipse
``{(a Du + b Dv) / 2 : a^2 + b^2 < 1}``. The reference drops degenerate photons
(``Du . (Dv x n) == 0``) by boolean-mask compaction, which synchronises with the host; here
they keep their slot with channel -1, which the splat kernels skip (zero contribution, zero
gradient), so shapes stay static and nothing waits on the device.
"""
import torch

from . import photon_differential
from ._lib import check, lib
from .photon_differential import PDS
from .splatting import SplatPlan, _cfg_ref, _on, _ptr, _stream

__all__ = ["change_of_basis_matrix", "splat_inputs", "splat_photons"]


def change_of_basis_matrix(Du, Dv, normal):
    """-> (Mp [2,3,N], good [N] bool). Degenerate photons get a finite placeholder."""
    tmp = torch.cross(Dv, normal, dim=0)
    den = (Du * tmp).sum(0)
    good = den != 0
    factor = 2.0 / torch.where(good, den, torch.ones_like(den))
    Mp = factor * torch.stack((tmp, torch.cross(normal, Du, dim=0)), dim=0)
    return Mp, good


def splat_inputs(Du, Dv, normal, flux, channel):
    """Splat inputs ``(Ep, Mp, cp, radius)`` for photons with receiver-plane differentials.

    ``Du, Dv, normal``: ``[3, N]``; ``flux``: ``[N]``; ``channel``: ``[N]`` int64.
    """
    Mp, good = change_of_basis_matrix(Du, Dv, normal)
    radius = 0.5 * torch.maximum(Du.norm(dim=0), Dv.norm(dim=0))
    area = torch.cross(Du, Dv, dim=0).norm(dim=0)
    Ep = flux / torch.where(good, area, torch.ones_like(area)) * 4
    cp = torch.where(good, channel, torch.full_like(channel, -1)).reshape(1, -1)
    return Ep.contiguous(), Mp.contiguous(), cp.contiguous(), radius.contiguous()


class _SplatPhotons(torch.autograd.Function):
    """``splat_inputs`` and the splat in one node: one kernel each way for the splat inputs
    (``pds_splat_inputs_f32``), the backward's reading the splat gradients as the plan's records.
    Plain float32 CUDA tensors only (``_fusable``)."""

    @staticmethod
    def forward(ctx, Du, Dv, normal, flux, xy, channel, output_size, max_pixel_radius):
        n, dev = flux.numel(), flux.device
        Ep, radius = torch.empty_like(flux), torch.empty_like(flux)
        Mp = torch.empty((2, 3, n), dtype=torch.float32, device=dev)
        cp = torch.empty((1, n), dtype=torch.int64, device=dev)
        with _on(dev):
            check(lib().pds_splat_inputs_f32(_ptr(Du), _ptr(Dv), _ptr(normal), _ptr(flux),
                                             _ptr(channel), n, _ptr(Ep), _ptr(Mp), _ptr(cp),
                                             _ptr(radius), _stream(dev)))
        plan, out = SplatPlan.splat((Ep, xy, Mp, cp, radius), output_size, max_pixel_radius)
        ctx.save_for_backward(Du, Dv, normal, flux, xy, channel, Ep, Mp, cp, radius)
        ctx.shape = (plan.C, plan.H, plan.W)
        ctx.mpr = plan.mpr
        ctx.cfg = plan.cfg
        ctx.plan_ws = plan.ws if photon_differential._keep_plan else None
        return out

    @staticmethod
    def backward(ctx, grad):
        Du, Dv, normal, flux, xy, channel, Ep, Mp, cp, radius = ctx.saved_tensors
        ws, ctx.plan_ws = ctx.plan_ws, None
        plan = SplatPlan.planned((Ep, xy, Mp, cp, radius), ctx.shape, ctx.mpr, ctx.cfg, ws)
        if torch.is_grad_enabled():  # create_graph: the splat inputs' own torch operations
            gE, gX, gM = plan.backward(grad.contiguous())
            # (views: the inputs' own hooks are run by the engine that asked for these gradients)
            real = [t.view_as(t) for t in (Du, Dv, normal, flux)]
            E, M, _, _ = splat_inputs(*real, channel)
            wanted = [t for t, w in zip(real, ctx.needs_input_grad) if w]
            # (E does not depend on the normal, nor M on the flux)
            outs = [(o, g) for o, g in ((E, gE), (M, gM)) if o.requires_grad]
            got = iter(torch.autograd.grad([o for o, _ in outs], wanted, [g for _, g in outs],
                                           create_graph=True, allow_unused=True) if wanted else ())
            grads = [next(got) if w else None for w in ctx.needs_input_grad[:4]]
            return (*grads, gX, None, None, None)
        plan.backward(grad.contiguous(), records=True)
        gX = torch.empty_like(xy)
        grads = [torch.empty_like(t) if w else None
                 for t, w in zip((Du, Dv, normal, flux), ctx.needs_input_grad)]
        with _on(flux.device):
            check(lib().pds_splat_inputs_backward_planned_f32(
                _ptr(Du), _ptr(Dv), _ptr(normal), _ptr(flux), flux.numel(), *ctx.shape,
                _ptr(plan.ws), plan.ws.numel(), _cfg_ref(ctx.cfg), _ptr(gX),
                *(_ptr(g) for g in grads), _stream(flux.device)))
        return (*grads, gX if ctx.needs_input_grad[4] else None, None, None, None)


def _fusable(Du, Dv, normal, flux, xy, channel):
    """Whether the kernels take these photons as they are: plain float32 CUDA tensors of one
    device, [3, N] each, [N] fluxes, an int64 [N] channel (anything else, broadcast shapes among
    it, goes through the torch operations)."""
    n = flux.numel()
    real = (Du, Dv, normal, flux, xy)
    return (n > 0 and flux.shape == (n,) and Du.shape == Dv.shape == normal.shape == (3, n) and
            xy.shape == (2, n) and channel.shape == (n,) and channel.dtype == torch.int64 and
            all(type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and
                t.device == flux.device for t in (*real, channel)) and
            all(t.dtype == torch.float32 for t in real))


def splat_photons(Du, Dv, normal, flux, positions_xy, channel, output_size, max_pixel_radius=20):
    """``model/caustics.py:233-239``: splat photons given their receiver-plane position
    ``positions_xy [2, N]`` (normalised receiver coordinates) and differentials."""
    if _fusable(Du, Dv, normal, flux, positions_xy, channel):
        return _SplatPhotons.apply(*(t.contiguous() for t in (Du, Dv, normal, flux, positions_xy,
                                                              channel)),
                                   tuple(output_size), max_pixel_radius)
    Ep, Mp, cp, radius = splat_inputs(Du, Dv, normal, flux, channel)
    return PDS.apply(Ep, positions_xy.contiguous(), Mp, cp, radius, tuple(output_size),
                     max_pixel_radius)
