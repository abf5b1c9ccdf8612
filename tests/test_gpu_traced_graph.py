"""``caustics.splat_photons`` with ``create_graph`` and a single input that requires a gradient: the
first gradient and, where it has a graph, its own gradient, as by the torch operations it stands for
(tolerances as in test_gpu_traced)."""
import pytest
import torch

from shapefromcaustics_b200 import caustics
from test_gpu_traced import by_torch, rel, traced

pytestmark = pytest.mark.gpu

NAMES = ["Du", "Dv", "normal", "flux", "xy"]


@pytest.mark.parametrize("wanted", [(k,) for k in range(5)] + [(3, 4), (2, 4), (2, 3)],
                         ids=lambda w: "+".join(NAMES[k] for k in w))
def test_some_inputs_with_a_graph(cuda, wanted):
    t = traced(300, zero=False)
    shape = (1, 64, 64)
    G = torch.randn(shape, generator=torch.Generator().manual_seed(92)).cuda()
    first, second = [], []
    for fn in (caustics.splat_photons, by_torch):
        x = [v.clone().requires_grad_(k in wanted) for k, v in enumerate(t[:5])]
        img = fn(*x, t[5], shape)
        leaves = [x[k] for k in wanted]
        g = torch.autograd.grad(img, leaves, G, create_graph=True)
        first.append(g)
        total = sum((v ** 2).sum() for v in g)
        second.append(torch.autograd.grad(total, leaves, allow_unused=True)
                      if total.requires_grad else [None] * len(leaves))
    for a, b in zip(*first):
        assert a.requires_grad == b.requires_grad
        assert rel(a, b) <= 1e-4
    for a, b in zip(*second):
        assert (a is None) == (b is None)
        if a is not None and float(b.abs().max()) > 0:
            assert rel(a, b) <= 1e-4
