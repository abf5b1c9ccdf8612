"""The forward where photons of very different energies share a screen tile: every pixel is right
for what covers it, not only for the brightest pixels of the image. Against the FP64 oracle, pixel by
pixel, the error is at most 1e-5 of the peaks (3/pi E) of the photons whose boxes hold the pixel, summed.

A photon evaluated in float32 is off by up to 2 (1 - s) ds of its peak, ds a few roundings of numbers
below 1 and of a coordinate below 20 px over a half-width of 0.5 px and more: 2e-6. Sums of at most a few
thousand such terms gather less than as much again."""
import math

import numpy as np
import pytest
import torch

from oracle import oracle as O
from shapefromcaustics_b200 import synthetic as S
from test_gpu_splat import run_gpu, to_np

pytestmark = pytest.mark.gpu

WALKS = [dict(), dict(walk=4), dict(walk=2), dict(coop_radius=3)]


def assert_every_pixel(photons, shape, cfg=None):
    img, _ = run_gpu(photons, shape, 20, S.upstream_grad(shape, seed=7), cfg)
    E, X, M, C, R = to_np(photons)
    ref = O.forward(E, X, M, C, R, shape, 20)
    peaks = O.forward(E, X, 0.0 * M, C, R, shape, 20)  # s = 0 all over each box
    assert bool(np.all(img[peaks == 0] == 0))
    worst = float(np.max(np.abs(img - ref)[peaks > 0] / peaks[peaks > 0]))
    assert worst <= 1e-5, worst


def round_photons(pos, s, e, H, W):
    n = pos.shape[1]
    s = torch.full((n,), float(s), dtype=torch.float64)
    return S.photons_from_pixels(pos, torch.zeros(n, dtype=torch.float64), s, s, e, H, W)


def two_bands(n, dim, each, seed=86, H=128, W=192):
    """n photons of energy 1 in the left half of every 64 px column of the image, and `each` photons
    of every energy in `dim` in the right half, out of their reach."""
    g = torch.Generator().manual_seed(seed)
    r = lambda k: torch.rand(k, generator=g, dtype=torch.float64)  # noqa: E731
    m = each * len(dim)
    x = torch.cat((4 + 24 * r(n), 40 + 18 * r(m))) + 64 * torch.randint(0, W // 64, (n + m,), generator=g)
    e = torch.cat((torch.ones(n), torch.tensor(dim).repeat(each))).double()
    order = torch.randperm(n + m, generator=g)
    return round_photons(torch.stack((x, H * r(n + m)))[:, order], 2.3, e[order], H, W)


@pytest.mark.parametrize("cfg", WALKS)
@pytest.mark.parametrize("n", [0, 300, 20000])
def test_dim_photons_beside_bright_ones(cuda, n, cfg):
    assert_every_pixel(two_bands(n, [1e-1, 1e-3, 1e-5, 1e-6, 1e-8], 40), (1, 128, 192), cfg)


def test_single_photons_beside_a_caustic(cuda):
    # work chunks of 2048 photons and more, nearly all of them on one spot
    g = torch.Generator().manual_seed(87)
    n, dim = 4_000_000, [1.0, 1e-2, 1e-4, 1e-6]
    E, X, M, C, R = two_bands(0, dim, 30, H=64, W=64)
    pos = torch.tensor([[12.3], [30.8]], dtype=torch.float64) + \
        torch.randn((2, n), generator=g, dtype=torch.float64)
    big = round_photons(pos, 1.5, 0.5 + 0.5 * torch.rand(n, generator=g, dtype=torch.float64), 64, 64)
    ph = [torch.cat((a, b), dim=-1) for a, b in zip((E, X, M, C, R), big)]
    assert_every_pixel(ph, (1, 64, 64))


@pytest.mark.parametrize("cfg", WALKS)
@pytest.mark.parametrize("n", [60, 2000, 30000])
def test_six_decades(cuda, n, cfg):
    E, X, M, C, R = S.uniform_cluster_photons(n, 130, 190, seed=88)
    g = torch.Generator().manual_seed(89)
    E = torch.exp(-math.log(1e6) * torch.rand(n, generator=g)).float()
    assert_every_pixel((E, X, M, C, R), (1, 130, 190), cfg)


@pytest.mark.parametrize("cfg", WALKS)
def test_energies_of_a_traced_caustic(cuda, cfg):
    # E by the inverse of the footprint's area, over three decades and more
    E, X, M, C, R = S.caustic_curve_photons(2 ** 17, 256, 256, seed=90, s_range=(0.5, 16.0))
    det = (M[0, 0] * M[1, 1] - M[0, 1] * M[1, 0]).abs()
    assert_every_pixel((E * det / det.max(), X, M, C, R), (1, 256, 256), cfg)
