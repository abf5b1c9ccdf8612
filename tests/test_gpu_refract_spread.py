"""The refraction backward on both sides of the field size that separates its two kernels (16384
texels), over photon orders that send its warps down each path: neighbouring texels (raster), one
2 x 2 block of cells (texel by texel; a warp on the border folds its patch), scattered (random),
and photon counts that leave partial warps. Tolerance as for the refraction backward elsewhere:
relative L2 below 1e-4 against float64 autograd; the orders differ among themselves by float32
sums only, below 1e-5."""
import numpy as np
import pytest
import torch

from oracle import refraction_chain as RF

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("H,W", [(127, 129), (128, 128), (64, 300)])
@pytest.mark.parametrize("per,cut", [(1, 0), (5, 13)])
def test_orders_and_field_sizes(cuda, H, W, per, cut):
    from shapefromcaustics_b200 import plate as PL
    scene = RF.PlateScene(texel=0.4, receiver_distance=30.0, receiver_half=0.25 * max(H, W))
    h = RF.height_field_bumps(H, W, seed=1, bumps=10, base=1.0, amp=(0.0, 0.05),
                              width=(2.0, 8.0)).float()
    ph = RF.jittered_photons(H, W, scene, per_texel=per, seed=2, smoothing=3.0)  # texel by texel
    n = ph[0].numel() - cut
    ph = [t[..., :n] for t in ph]
    params = PL.plate_params(scene, float(ph[2][0, 0]))
    g = torch.Generator().manual_seed(0)
    gE, gX = torch.randn(n, generator=g).double(), torch.randn((2, n), generator=g).double()
    gM = 1e-3 * torch.randn((2, 3, n), generator=g).double()
    gM[:, 2] = 0
    h64 = h.double().requires_grad_(True)
    px, py, flux = (t.float() for t in (ph[0], ph[1], ph[4]))
    Ep, xp, Mp, _, _ = RF.receiver_splat_inputs(h64, scene, (px.double(), py.double(), ph[2].double(),
                                                             ph[3].double(), flux.double()))
    ((Ep * gE).sum() + (xp * gX).sum() + (Mp * gM).sum()).backward()
    raster = torch.argsort(torch.arange(n) % per, stable=True)
    got = []
    for order in (torch.arange(n), raster, torch.randperm(n, generator=g)):
        dev = [t[..., order].float().contiguous().cuda() for t in (px, py, flux, gE, gX, gM)]
        got.append(PL.refract_backward(h.cuda(), *dev[:3], params, *dev[3:]).cpu())
        assert rel_l2(got[-1], h64.grad) < 1e-4
        assert rel_l2(got[-1], got[0]) < 1e-5
