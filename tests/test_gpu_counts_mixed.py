"""The forward's accumulator where one segment mixes photons that its walks treat differently,
against the FP64 oracle at the forward's tolerance (relative L2 <= 1e-5): photons gathered on a few
pixels, four million of them, so that a work chunk is large enough for its counts to wrap, half of
them with a band and half without (a support wider than the radius limit's box, a radius below the
support's) or splatted by their whole warp."""
import math

import pytest
import torch

from shapefromcaustics_b200 import synthetic as S
from test_gpu_splat import assert_parity

pytestmark = pytest.mark.gpu

N = 4_000_000  # chunks of 2048 photons and more (148 SMs, twelve chunks each)


def gathered(s, seed=85, n=N, H=70, W=83):
    """n photons within 0.02 px of a point between pixels; photon i has semi-axes s[i % 2] and 0.7
    of it (px)."""
    g = torch.Generator().manual_seed(seed)
    pos = torch.tensor([[33.4], [29.7]], dtype=torch.float64) + \
        0.02 * torch.randn((2, n), generator=g, dtype=torch.float64)
    theta = torch.rand(n, generator=g, dtype=torch.float64) * math.pi
    odd = torch.arange(n) % 2 == 1
    s1 = torch.where(odd, float(s[1]), float(s[0])).double()
    e = 0.5 + 0.5 * torch.rand(n, generator=g, dtype=torch.float64)
    return S.photons_from_pixels(pos, theta, s1, 0.7 * s1, e, H, W)


@pytest.mark.parametrize("class_bits", [5, -1])
@pytest.mark.parametrize("mpr", [1, 2, 3])
def test_supports_wider_than_the_limit(cuda, mpr, class_bits):
    # the second kind's support is several times its box: no band
    assert_parity(gathered((1.2 * mpr, 4.0 * mpr)), (1, 70, 83), mpr,
                  cfg=dict(class_bits=class_bits))


@pytest.mark.parametrize("class_bits", [5, -1])
def test_radius_below_the_support(cuda, class_bits):
    E, X, M, C, R = gathered((5.0, 5.0))
    R = torch.where(torch.arange(N) % 2 == 1, 0.3 * R, R)
    assert_parity((E, X, M, C, R), (1, 70, 83), 20, cfg=dict(class_bits=class_bits))


@pytest.mark.parametrize("cfg", [dict(coop_radius=8), dict(coop_radius=8, walk=4),
                                 dict(coop_radius=3, tile=32)])
def test_whole_warp_photons(cuda, cfg):
    assert_parity(gathered((1.0, 10.0)), (1, 70, 83), 20, cfg=dict(class_bits=-1, **cfg))
