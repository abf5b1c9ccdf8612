"""``caustics.splat_photons`` on the fused kernels (plain float32 CUDA tensors) against the torch
operations it stands for (``splat_inputs`` and ``PDS``), and what the fused path leaves to them.

Tolerances: the image and the gradients are float32 evaluations of the same formulas, a few dozen
roundings of numbers that cancel by at most the photons' aspect ratio (16 here) and cross product
(64): 1e-5 and 1e-4 relative L2, the splat's own against float64."""
import pytest
import torch

from shapefromcaustics_b200 import PDS
from shapefromcaustics_b200 import caustics

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-300))


def traced(n, seed=90, zero=True):
    """Differentials of 0.01..0.16 in receiver units about a tilted receiver normal, some
    degenerate (parallel or zero differentials), some off the image, some of other channels."""
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.rand(s, generator=g)  # noqa: E731
    th = 6.28 * r(n)
    s1, s2 = 0.01 * 16 ** r(n), 0.01 * 16 ** r(n)
    Du = torch.stack((s1 * th.cos(), s1 * th.sin(), 0.02 * s1))
    Dv = torch.stack((-s2 * th.sin(), s2 * th.cos(), 0.01 * s2))
    if zero and n > 8:
        Du[:, 3] = 0.0
        Dv[:, 5] = 0.0
    nrm = torch.zeros(3, n)
    nrm[2], nrm[0] = 1.0, 0.05
    t = [Du, Dv, nrm, 1e-3 * (0.5 + r(n)), 2.4 * r(2, n) - 1.2, torch.randint(-1, 3, (n,), generator=g)]
    return [x.cuda() for x in t]


def run(fn, t, shape, grad, create_graph=False):
    leaves = [x.clone().requires_grad_(True) for x in t[:5]]
    img = fn(*leaves, t[5], shape)
    return img, leaves, torch.autograd.grad(img, leaves, grad, create_graph=create_graph)


def by_torch(Du, Dv, normal, flux, xy, channel, shape):
    Ep, Mp, cp, radius = caustics.splat_inputs(Du, Dv, normal, flux, channel)
    return PDS.apply(Ep, xy.contiguous(), Mp, cp, radius, shape, 20)


@pytest.mark.parametrize("n", [1, 255, 256, 257, 20011])
@pytest.mark.parametrize("shape", [(1, 64, 64), (2, 75, 131)])
def test_fused_equals_the_torch_operations(cuda, n, shape):
    t = traced(n)
    grad = torch.randn(shape, generator=torch.Generator().manual_seed(91)).cuda()
    img, _, got = run(caustics.splat_photons, t, shape, grad)
    ref, _, want = run(by_torch, t, shape, grad)
    assert type(img.grad_fn).__name__ == "_SplatPhotonsBackward"
    assert rel(img, ref) <= 1e-5
    for a, b in zip(got, want):
        assert a.shape == b.shape and bool(torch.isfinite(a).all())
        assert rel(a, b) <= 1e-4 or float((a - b).abs().max()) <= 1e-12


def test_what_the_fused_path_does_not_take(cuda):
    n, shape = 500, (1, 64, 64)
    Du, Dv, nrm, flux, xy, ch = traced(n)
    ref = by_torch(Du, Dv, nrm, flux, xy, ch, shape)
    wide = torch.stack((Du, Du), dim=-1)[..., 0]  # not contiguous: copied, still fused
    assert not wide.is_contiguous()
    assert rel(caustics.splat_photons(wide, Dv, nrm, flux, xy, ch, shape), ref) <= 1e-5
    # a broadcast channel goes through the torch operations
    one = torch.zeros(1, dtype=torch.int64, device="cuda")
    got = caustics.splat_photons(Du, Dv, nrm, flux, xy, one, shape)
    assert rel(got, by_torch(Du, Dv, nrm, flux, xy, torch.zeros_like(ch), shape)) <= 1e-5
    # and what they refuse is refused with their message
    with pytest.raises(RuntimeError, match="expected scalar type Long"):
        caustics.splat_photons(Du, Dv, nrm, flux, xy, ch.int(), shape)
    with pytest.raises(RuntimeError, match="float32"):
        caustics.splat_photons(*(x.double() for x in (Du, Dv, nrm, flux, xy)), ch, shape)


def test_gradients_with_a_graph_keep_the_inputs_operations(cuda):
    t = traced(300, zero=False)
    shape = (1, 64, 64)
    grad = torch.ones(shape, device="cuda")
    out = []
    for fn in (caustics.splat_photons, by_torch):
        _, leaves, g = run(fn, t, shape, grad, create_graph=True)
        out.append(torch.autograd.grad((g[0] ** 2).sum(), leaves[0])[0])
    assert rel(*out) <= 1e-4
