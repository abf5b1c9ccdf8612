"""The batched plates' refraction backward on fields large enough for the kernel without patch
regions (16384 texels and more), at photon counts that leave partial and empty warps in its last
CTA of 64, by gradient arrays and by the splat plan's records, in texel and in raster order (a
warp's photons in one 2 x 2 block of cells, or along a row): the height gradient against the sum of
the simulations' own plates. The same photons' float32 gradients in another order of summation:
relative L2 below 1e-5, as for the batch on smaller fields."""
import pytest
import torch

from oracle import refraction_chain as RF

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-300))


def plates(H, W, residue, order):
    """Three simulations of one field, their photon counts' sum congruent to residue mod 64."""
    from shapefromcaustics_b200 import plate as PL
    half = 0.25 * max(H, W)
    h = RF.height_field_bumps(H, W, seed=1, bumps=10, base=1.0, amp=(0.0, 0.05),
                              width=(2.0, 8.0)).float().cuda()
    sims, photons, total = [], [], 0
    for k, (per, image) in enumerate([(1, 64), (3, 96), (40, 64)]):
        scene = RF.PlateScene(texel=0.4 + 0.05 * k, receiver_distance=30.0, receiver_half=half)
        ph = RF.jittered_photons(H, W, scene, per_texel=per, seed=2 + k, smoothing=3.0)
        px, py, flux = (t.float() for t in (ph[0], ph[1], ph[4]))
        n = px.numel()
        if order == "raster":
            by = torch.argsort(torch.arange(n) % per, stable=True)
            px, py, flux = px[by], py[by], flux[by]
        if k == 2:
            n -= (total + n - residue) % 64
        total += n
        photons.append([t[:n].contiguous().cuda() for t in (px, py, flux)])
        sims.append((n, (1, image, image), PL.plate_params(scene, float(ph[2][0, 0]))))
    assert total % 64 == residue
    return h, sims, photons


@pytest.mark.parametrize("residue", [0, 1, 2, 31, 32, 33, 63])
@pytest.mark.parametrize("H,W", [(128, 128), (131, 150)])
@pytest.mark.parametrize("order", ["texel", "raster"])
def test_partial_warps(cuda, residue, H, W, order):
    from shapefromcaustics_b200 import plate as PL
    from shapefromcaustics_b200._lib import check, lib
    from shapefromcaustics_b200.splatting import _ptr, _stream
    h, sims, photons = plates(H, W, residue, order)
    batch = PL.BatchedPlate(sims, 20, "cuda")
    cat = [torch.cat([p[k] for p in photons]).contiguous() for k in range(3)]
    g = torch.Generator("cuda").manual_seed(3)
    # by records
    flat = batch.forward(h, *cat)
    G = torch.randn(flat.shape, generator=g, device="cuda")
    got = batch.backward(h, *cat, G)
    want, off = torch.zeros_like(h), 0
    for (n, shape, p), ph in zip(sims, photons):
        hs = h.clone().requires_grad_(True)
        size = shape[1] * shape[2]
        image = PL.PlateSplat.apply(hs, *ph, p, shape, 20, True)
        image.backward(G[off:off + size].view(shape))
        want += hs.grad
        off += size
    assert bool(torch.isfinite(got).all())
    assert rel_l2(got, want) < 1e-5
    # by arrays
    n = batch.n_total
    gE, gX = (torch.randn(s, generator=g, device="cuda") for s in ((n,), (2, n)))
    gM = 1e-3 * torch.randn((2, 3, n), generator=g, device="cuda")
    got = torch.zeros_like(h)
    with torch.cuda.device(h.device):
        check(lib().pds_batch_refract_backward_f32(
            _ptr(h), H, W, _ptr(batch.plates_dev), _ptr(batch.begins_dev), batch.n_sims,
            *(_ptr(t) for t in cat), n, _ptr(gE), _ptr(gX), _ptr(gM), _ptr(got),
            _stream(h.device)))
    want, off = torch.zeros_like(h), 0
    for (m, _, p), ph in zip(sims, photons):
        own = [t[..., off:off + m].contiguous() for t in (gE, gX, gM)]
        PL.refract_backward(h, *ph, p, *own, want)
        off += m
    assert bool(torch.isfinite(got).all())
    assert rel_l2(got, want) < 1e-5
