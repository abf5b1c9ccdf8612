"""The plan's binning where its shape changes: photon counts around one plan CTA, bucket counts
around the limits of the place pass's own scan (4608) and of the one-kernel scan (131072), and
beyond (three scan kernels); each against the CPU restatement of the binning. A plan's forward
and backward run twice give the same results: the tile kernels leave their work counters at
zero, and wide footprints are splatted by the tile kernels' own CTAs."""
import pytest
import torch

from oracle import plan_keys as PK
from shapefromcaustics_b200 import _lib
from shapefromcaustics_b200 import synthetic as S
from shapefromcaustics_b200.splatting import SplatPlan
from test_gpu_plan import check_binning, export

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 767, 768, 769, 30011])
@pytest.mark.parametrize("H,W", [(64, 64), (768, 768), (780, 768), (4096, 4096), (4160, 4096)])
def test_binning_at_the_scan_limits(cuda, n, H, W):
    ph = S.uniform_cluster_photons(n, H, W, seed=60 + n, s_range=(0.3, 9.0))
    cfg = _lib.config(apron_max=6)  # footprints wider than 6 px take the wide list
    plan = SplatPlan(*(t.cuda() for t in ph), (1, H, W), 20, config=cfg)
    n_tiles = ((H + 63) // 64) * ((W + 63) // 64)
    kg, sl = export(plan.ws, n, n_tiles, 20, cfg)
    kc, _ = PK.plan_keys([t.numpy() for t in ph], [(n, (1, H, W))], 20, apron_max=6, class_bits=5)
    check_binning(kg, sl, kc, n_tiles, 5)


@pytest.mark.parametrize("walk", [3, 4])
def test_a_plan_serves_several_passes(cuda, walk):
    n, H, W = 50021, 200, 300
    ph = [t.cuda() for t in S.uniform_cluster_photons(n, H, W, seed=70, s_range=(0.3, 9.0))]
    g = S.upstream_grad((1, H, W), seed=71).cuda()
    plan = SplatPlan(*ph, (1, H, W), 20, config=_lib.config(apron_max=6, walk=walk))
    imgs = [plan.forward() for _ in range(2)]
    grads = [plan.backward(g) for _ in range(2)]
    # the same photons' float32 sums in another order: each pixel's rounding is at most
    # (adds a pixel, here below 2^8) * 2^-24 of it
    assert torch.allclose(imgs[0], imgs[1], rtol=2.0 ** -16, atol=0)
    for a, b in zip(*grads):
        assert torch.equal(a, b)
    full = SplatPlan(*ph, (1, H, W), 20).forward()  # no wide list
    assert torch.allclose(imgs[0], full, rtol=1e-4, atol=1e-5 * float(full.abs().max()))
