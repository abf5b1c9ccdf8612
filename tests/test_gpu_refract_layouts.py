"""The refraction backwards on gradients that are not contiguous: their copies live until the kernel
that reads them is enqueued (three copies of one call, none in another's memory). Against the same
call on contiguous gradients: only the order of the float sums into the field differs (1e-5)."""
import pytest
import torch

from oracle import refraction_chain as RF
from test_gpu_plate import point_scene, rel_l2

pytestmark = pytest.mark.gpu


def strided(n, seed=21):
    """d L / d (Ep, xp, Mp) of n photons, every second element of larger tensors."""
    g = torch.Generator("cuda").manual_seed(seed)
    scales = ((), 1.0), ((2,), 1.0), ((2, 3), 1e-3)
    return [(k * torch.randn((*s, 2 * n), generator=g, device="cuda"))[..., ::2] for s, k in scales]


@pytest.mark.parametrize("per", [1, 4, 30])
def test_collimated(cuda, per):
    from shapefromcaustics_b200 import plate as PL
    scene = RF.PlateScene(texel=0.4, receiver_distance=30.0, receiver_half=12.0)
    h = RF.height_field_bumps(48, 48, seed=1, bumps=10, base=1.0, amp=(0.0, 0.05),
                              width=(2.0, 8.0)).float().cuda()
    ph = RF.jittered_photons(48, 48, scene, per_texel=per, seed=2, smoothing=3.0)
    px, py, flux = (t.float().cuda() for t in (ph[0], ph[1], ph[4]))
    params = PL.plate_params(scene, float(ph[2][0, 0]))
    grads = strided(px.numel())
    assert not any(t.is_contiguous() for t in grads)
    got = PL.refract_backward(h, px, py, flux, params, *grads)
    held = [t.contiguous() for t in grads]
    want = PL.refract_backward(h, px, py, flux, params, *held)
    assert rel_l2(got.cpu(), want.cpu()) < 1e-5


@pytest.mark.parametrize("n_dir", [2000, 60000])
def test_point_light(cuda, n_dir):
    from shapefromcaustics_b200 import plate as PL
    scene, h, light, (d, dt, dp, flux) = point_scene(n_dir=n_dir, seed=3)
    params = PL.plate_params(scene, 0.0)
    grads = strided(flux.numel())
    got = PL.refract_point_backward(h.cuda(), light, params, d, dt, dp, flux, *grads)
    held = [t.contiguous() for t in grads]
    want = PL.refract_point_backward(h.cuda(), light, params, d, dt, dp, flux, *held)
    assert rel_l2(got.cpu(), want.cpu()) < 1e-5
