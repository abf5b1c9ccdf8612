"""The point-light backward adds patch rows as aligned 16-byte reductions: every alignment of the
field's rows (odd widths, a gradient that starts at any float of its buffer), patches folded at the
border, fields of a few texels, the buffer's first and last quads (its neighbours stay untouched),
and the gradients as arrays or as the plan's records. Tolerances as for the point-light backward
elsewhere (relative L2 below 1e-3 against float64 autograd); the same photons' sums differ among
alignments and modes by the order of float32 additions, below 1e-5."""
import numpy as np
import pytest
import torch

from oracle import refraction_chain as RF

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def point_photons(H, W, n_dir):
    from shapefromcaustics_b200 import plate as PL
    scene = RF.PlateScene(texel=0.4, receiver_distance=30.0, receiver_half=0.25 * max(H, W))
    h = RF.height_field_bumps(H, W, seed=1, bumps=4, base=1.0, amp=(0.0, 0.05),
                              width=(2.0, 8.0)).float()
    hx, hy = 0.49 * 0.4 * (W - 1), 0.49 * 0.4 * (H - 1)
    light = PL.point_light((0.5, -0.4, 40.0), (-hx, -hy, hx, hy), 1.0, 3.0, 1.0)
    d, dt, dp, flux, _ = PL.point_light_source(light, n_dir, "cuda", seed=4)
    return scene, h, light, d, dt, dp, flux


@pytest.mark.parametrize("H,W", [(3, 4), (4, 3), (5, 5), (9, 31), (48, 49), (33, 64)])
def test_alignments(cuda, H, W):
    from shapefromcaustics_b200 import plate as PL
    scene, h, light, d, dt, dp, flux = point_photons(H, W, 3001)
    params = PL.plate_params(scene, 0.0)
    n = flux.numel()
    g = torch.Generator().manual_seed(0)
    gE, gX = torch.randn(n, generator=g).double(), torch.randn((2, n), generator=g).double()
    gM = 1e-3 * torch.randn((2, 3, n), generator=g).double()
    gM[:, 2] = 0
    h64 = h.double().requires_grad_(True)
    Ep, xp, Mp, _, _ = RF.point_light_splat_inputs(
        h64, scene, tuple(light.position), d.double().cpu(), dt.double().cpu(), dp.double().cpu(),
        flux.double().cpu(), float(light.plane_z))
    ((Ep * gE).sum() + (xp * gX).sum() + (Mp * gM).sum()).backward()
    dev = [t.float().cuda() for t in (gE, gX, gM)]
    first = None
    for off in range(4):
        buf = torch.zeros(H * W + 8, device="cuda")
        view = buf[off:off + H * W].view(H, W)
        PL.refract_point_backward(h.cuda(), light, params, d, dt, dp, flux, *dev, grad_height=view)
        first = view.cpu() if off == 0 else first
        assert rel_l2(view.cpu(), h64.grad) < 1e-3
        assert rel_l2(view.cpu(), first) < 1e-5
        assert not buf[:off].any() and not buf[off + H * W:].any()


@pytest.mark.parametrize("H,W", [(9, 31), (48, 49)])
def test_records_equal_arrays(cuda, H, W):
    from shapefromcaustics_b200 import plate as PL
    from shapefromcaustics_b200.splatting import SplatPlan
    scene, h, light, *photons = point_photons(H, W, 5000)
    params, shape = PL.plate_params(scene, 0.0), (1, 40, 52)
    G = torch.randn(shape, generator=torch.Generator().manual_seed(1)).cuda()
    plan = SplatPlan(*PL.refract_point_forward(h.cuda(), light, params, *photons), shape, 12)
    img = plan.forward()
    want = PL.refract_point_backward(h.cuda(), light, params, *photons, *plan.backward(G)).cpu()
    for keep in (True, False):
        hv = h.cuda().requires_grad_(True)
        got = PL.PointPlateSplat.apply(hv, *photons, light, params, shape, 12, keep)
        got.backward(G, retain_graph=True)
        assert rel_l2(got.detach().cpu(), img.cpu()) < 1e-5
        assert rel_l2(hv.grad.cpu(), want) < 1e-5
        got.backward(G)  # a second pass plans again
        assert rel_l2(hv.grad.cpu(), 2 * want) < 1e-5
