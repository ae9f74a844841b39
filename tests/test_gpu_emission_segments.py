"""The emission's row segments (their number grows with the Gaussians and views
of a launch) do not show in the images: batches against one view per call."""
import numpy as np
import pytest
import torch

import dmgs_gb300
from dmgs_gb300.batched import BatchedRasterizer
from dmgs_gb300.scenes import random_inside_view
from test_gpu_batched import D, _settings

pytestmark = pytest.mark.gpu


# 7, 9, 12 and 18 segments a row of 4 views of 100 tile rows on 152 SMs; single views have up to 32
@pytest.mark.parametrize("P", [300_000, 1_050_000, 2_100_000, 5_000_000])
def test_images_at_several_segment_counts(P):
    gen = torch.Generator(device=D).manual_seed(P)
    g = {"means3D": 2 * torch.rand(P, 3, device=D, generator=gen) - 1,
         "opacities": 0.3 * torch.rand(P, 1, device=D, generator=gen),
         "colors_precomp": torch.rand(P, 3, device=D, generator=gen),
         "scales": (0.002 + 0.01 * torch.rand(P, 3, device=D, generator=gen)) * (3e5 / P) ** (1 / 3),
         "rotations": torch.nn.functional.normalize(torch.randn(P, 4, device=D, generator=gen))}
    rng = np.random.default_rng(6)
    settings = [_settings(random_inside_view(rng, 200 - 8 * i, 1600 - i), deg=0) for i in range(4)]
    br = BatchedRasterizer(settings, g)
    br.forward()
    torch.cuda.synchronize()
    br.status()
    for v, rs in enumerate(settings):
        img = dmgs_gb300.GaussianRasterizer(rs)(means2D=torch.zeros_like(g["means3D"]), **g)[0]
        assert torch.equal(br.images[v], img), v
