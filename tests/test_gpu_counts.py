"""The forward's fixed-point accumulator where it can go wrong, against the FP64 oracle at the
forward's tolerance (relative L2 <= 1e-5): counts that wrap (photons gathered on few pixels, in
every walk), photons far brighter than the rest (added directly), energies near the ends of the
float range, and band rows cut by the box (a radius below the support's, the image's edges, the
radius limit) to odd widths."""
import pytest
import torch

from shapefromcaustics_b200 import synthetic as S
from test_gpu_splat import assert_parity

pytestmark = pytest.mark.gpu


def gathered(n, H, W, s, spread=0.01, seed=80):
    """n photons of s pixels within `spread` pixels of the image's centre."""
    g = torch.Generator().manual_seed(seed)
    pos = torch.tensor([[W / 2.0], [H / 2.0]]) + spread * torch.randn((2, n), generator=g,
                                                                     dtype=torch.float64)
    theta = torch.rand(n, generator=g, dtype=torch.float64) * 3.14
    one = torch.ones(n, dtype=torch.float64)
    return S.photons_from_pixels(pos, theta, s * one, 0.6 * s * one, 0.75 * one, H, W)


@pytest.mark.parametrize("cfg", [dict(), dict(walk=1), dict(walk=2), dict(walk=4),
                                 dict(coop_radius=2), dict(chunk=16384), dict(tile=16)])
@pytest.mark.parametrize("s,spread", [(0.8, 0.01), (6.0, 0.01), (6.0, 3.0)])
def test_gathered_photons(cuda, cfg, s, spread):
    assert_parity(gathered(9000, 90, 131, s, spread), (1, 90, 131), 20, cfg=cfg)


@pytest.mark.parametrize("walk", [3, 4])
def test_a_few_bright_photons(cuda, walk):
    E, X, M, C, R = S.uniform_cluster_photons(30000, 150, 200, seed=81)
    E = E.clone()
    E[::97] *= 3e4
    E[5] = 0.0
    assert_parity((E, X, M, C, R), (1, 150, 200), 20, cfg=dict(walk=walk))


@pytest.mark.parametrize("scale", [1e-33, 1e-20, 1e25, 1e33])
def test_extreme_energies(cuda, scale):
    E, X, M, C, R = S.uniform_cluster_photons(20000, 150, 200, seed=82)
    assert_parity((E * scale, X, M, C, R), (1, 150, 200), 20, grad_tol=1e-4)


@pytest.mark.parametrize("mpr", [0, 1, 2, 3, 20])
@pytest.mark.parametrize("H,W", [(33, 47), (64, 65), (130, 129)])
def test_rows_cut_by_the_box(cuda, H, W, mpr):
    E, X, M, C, R = S.uniform_cluster_photons(20011, H, W, seed=83 + mpr, s_range=(0.5, 5.0))
    assert_parity((E, X, M, C, 0.4 * R), (1, H, W), mpr)  # boxes inside the supports
    assert_parity((E, X, M, C, R), (1, H, W), mpr)
