"""Photons so thin that their band's half-width is lost in the rounding of a pixel coordinate, on
pixel corners, where pixels lie exactly on their centre line (s there is the offset along the line
alone): the forward and grad_Ep of the default walk, against the FP64 oracle at the forward's
tolerance (relative L2 <= 1e-5). The image's sides are powers of two and the slopes 0, infinity and +-1,
so that the centre line's pixels are exact in float32 too."""
import math

import numpy as np
import pytest
import torch

from shapefromcaustics_b200 import synthetic as S
from test_gpu_splat import rel_l2, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def thin(width, length=18.0, size=64, angles=(0.0, 0.25, 0.5, 0.75)):
    """Photons on pixel corners 3 px apart, of half-width `width` px across the direction
    `angle` pi, `length` px along it."""
    p = torch.arange(1.0, size, 3.0, dtype=torch.float64)
    y, x = torch.meshgrid(p, p, indexing="ij")
    n = x.numel()
    k = torch.arange(n) % len(angles)
    along = torch.tensor([[round(math.cos(math.pi * a), 12), round(math.sin(math.pi * a), 12)]
                          for a in angles], dtype=torch.float64)[k].T
    M = torch.zeros((2, 3, n), dtype=torch.float64)
    M[0, 0], M[0, 1] = -along[1] / width * (size / 2), along[0] / width * (size / 2)
    M[1, 0], M[1, 1] = along[0] / length * (size / 2), along[1] / length * (size / 2)
    xp = 2.0 * torch.stack((x.reshape(-1), y.reshape(-1))) / size - 1.0
    e = 0.5 + (torch.arange(n) % 7) / 14.0
    return (e.float(), xp.float(), M.float(), torch.zeros((1, n), dtype=torch.int64),
            torch.full((n,), 2.0 * length / size))


@pytest.mark.parametrize("width", [1e-9, 1e-8, 1e-7, 3e-7, 1e-6, 1e-5, 1e-3, 0.1])
def test_pixels_on_the_centre_line(cuda, width):
    ph, shape = thin(width), (1, 64, 64)
    grad = S.upstream_grad(shape, seed=9)
    img, g = run_gpu(ph, shape, 20, grad)
    rimg, r = run_oracle(ph, shape, 20, grad)
    assert np.count_nonzero(rimg) > 1000
    assert rel_l2(img, rimg) <= 1e-5
    assert rel_l2(g[0], r[0]) <= 1e-5
