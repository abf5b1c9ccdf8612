"""Autograd face of the splatting op: ``PDS``, with the reference's signature.

Mirror of ``model/photon_differential.py:7-19``: ``PDS.apply(Ep, xp, Mp, cp, radius,
output_size, max_pixel_radius)`` returns the ``[C,H,W]`` photon map and its backward returns
``(grad_Ep, grad_xp, grad_Mp, None, None, None, None)``.

Difference from the reference: the forward's photon binning and sort (the plan) is kept for
the backward instead of being recomputed. ``set_keep_plan(False)`` drops it after the forward
and rebuilds it in the backward, trading one binning pass for the plan's workspace (about 76
bytes per photon) held between the passes.
"""
import torch

from .splatting import SplatPlan, _check_photons

_keep_plan = True


def set_keep_plan(keep: bool):
    global _keep_plan
    _keep_plan = bool(keep)


class PDS(torch.autograd.Function):
    @staticmethod
    def forward(ctx, Ep, xp, Mp, cp, radius, output_size, max_pixel_radius):
        _check_photons(Ep, xp, Mp, cp, radius)
        plan, out = SplatPlan.splat((Ep, xp, Mp, cp, radius), output_size, max_pixel_radius)
        ctx.save_for_backward(Ep, xp, Mp, cp, radius)
        ctx.output_size = (plan.C, plan.H, plan.W)
        ctx.max_pixel_radius = plan.mpr
        ctx.plan_ws = plan.ws if _keep_plan else None
        ctx.cfg = plan.cfg
        return out

    @staticmethod
    def backward(ctx, grad_pds):
        Ep, xp, Mp, cp, radius = ctx.saved_tensors
        plan = SplatPlan.planned((Ep, xp, Mp, cp, radius), ctx.output_size, ctx.max_pixel_radius,
                                 ctx.cfg, ctx.plan_ws)
        grad_Ep, grad_xp, grad_Mp = plan.backward(grad_pds.contiguous())
        ctx.plan_ws = None
        return grad_Ep, grad_xp, grad_Mp, None, None, None, None
