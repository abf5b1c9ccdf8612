"""Tensor hooks on the inputs of ``caustics.splat_photons`` run once for a gradient, with and without
``create_graph``, as by the torch operations it stands for (tolerance as in test_gpu_traced)."""
import pytest
import torch

from shapefromcaustics_b200 import caustics
from test_gpu_traced import by_torch, rel, traced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("create_graph", [False, True])
def test_hooks_run_once(cuda, create_graph):
    t = traced(300, zero=False)
    shape = (1, 64, 64)
    G = torch.randn(shape, generator=torch.Generator().manual_seed(93)).cuda()
    got = []
    for fn in (caustics.splat_photons, by_torch):
        leaves = [v.clone().requires_grad_(True) for v in t[:5]]
        calls = [0] * 5

        def hook(k):
            def run(g):
                calls[k] += 1
                return 2 * g
            return run

        for k, v in enumerate(leaves):
            v.register_hook(hook(k))
        got.append(torch.autograd.grad(fn(*leaves, t[5], shape), leaves, G,
                                       create_graph=create_graph))
        assert calls == [1] * 5
    for a, b in zip(*got):
        assert rel(a, b) <= 1e-4
