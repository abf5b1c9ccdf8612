"""The projected update's volume heuristic at the edges of its tiles (64 x 16 pixels) and on both
sides of the largest box radius that the tile kernel takes (8), against the reference's operations
in float64. Each pixel is its own value plus mask * mean * factor: a few dozen float32 roundings of
numbers below the field's largest, so within 2^-18 of that (64 roundings of 2^-24)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [0, 1, 2, 8, 9])
@pytest.mark.parametrize("H,W", [(1, 1), (3, 200), (16, 64), (17, 65), (33, 63), (129, 300)])
@pytest.mark.parametrize("vol", ["below", "above", "inside"])
def test_update_at_the_tile_edges(cuda, H, W, radius, vol):
    from oracle.landweber_ref import landweber_update_reference
    from shapefromcaustics_b200.landweber import LandweberParams, landweber_update
    g = torch.Generator().manual_seed(H * 1000 + W + radius)
    d = 0.05 + 0.1 * torch.rand((H, W), generator=g)
    grad = torch.randn((H, W), generator=g)
    mask = (torch.rand((H, W), generator=g) > 0.1).float()
    v = float(d.sum())
    d1, d2 = {"below": (2 * v, 3 * v), "above": (0.1 * v, 0.6 * v), "inside": (0.1 * v, 3 * v)}[vol]
    p = LandweberParams(tau=1e-4, d1=d1, d2=d2, radius=radius)
    ref = landweber_update_reference(d.double(), grad.double(), mask.double(), p)
    out = landweber_update(d.cuda(), grad.cuda(), mask.cuda(), p).cpu().double()
    assert float((out - ref).abs().max()) <= 2.0 ** -18 * 0.3
