"""The batched forms by SH row length and alignment (float4 rows or not), and
by the number of Gaussians at which the emission's row segments change,
against one view per call."""
import numpy as np
import pytest
import torch

import dmgs_gb300
from dmgs_gb300.batched import BatchedRasterizer
from dmgs_gb300.scenes import random_inside_view
from helpers import rel_l2
from test_gpu_batched import D, _gauss, _plain, _scene_and_views, _settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coeffs,degree,offset", [(1, 0, 0), (4, 1, 0), (9, 2, 0), (12, 2, 0), (16, 3, 0), (16, 1, 0),
                                                  (16, 3, 1), (20, 3, 0)])
@pytest.mark.parametrize("P", [127, 3000])
def test_gradients_by_row_length_and_alignment(coeffs, degree, offset, P):
    sc, views = _scene_and_views(P=P, seed=47)
    g = _gauss(sc)
    rows = torch.zeros(P, 20, 3, device=D)
    rows[:, :16] = g["shs"]
    flat = torch.empty(P * coeffs * 3 + offset, device=D)
    g["shs"] = flat[offset:].view(P, coeffs, 3)
    g["shs"].copy_(rows[:, :coeffs])
    settings = [_settings(v, deg=degree) for v in views]
    gen = torch.Generator(device=D).manual_seed(3)
    dimgs = [torch.randn(3, v.height, v.width, device=D, generator=gen) for v in views]
    plain = [_plain(g, rs, d) for rs, d in zip(settings, dimgs)]
    br = BatchedRasterizer(settings, g)
    br.forward()
    br.backward(dimgs)
    torch.cuda.synchronize()
    br.status()
    for v in range(len(views)):
        assert torch.equal(br.images[v], plain[v][0])
    for k in g:
        want = sum(p[1][k] for p in plain)
        assert rel_l2(br.grads[k].cpu().numpy(), want.cpu().numpy()) <= 1e-5, k
    assert not br.grads["shs"][:, (degree + 1) ** 2:].any()


@pytest.mark.parametrize("P", [(1 << 20) - 1, 1 << 20])
def test_images_on_both_sides_of_the_segment_rule(P):
    """16 views: 16 x 2^20 Gaussians is where the rule changes."""
    gen = torch.Generator(device=D).manual_seed(9)
    g = {"means3D": 2 * torch.rand(P, 3, device=D, generator=gen) - 1,
         "opacities": torch.rand(P, 1, device=D, generator=gen),
         "shs": torch.randn(P, 1, 3, device=D, generator=gen),
         "scales": 0.002 + 0.01 * torch.rand(P, 3, device=D, generator=gen),
         "rotations": torch.nn.functional.normalize(torch.randn(P, 4, device=D, generator=gen))}
    rng = np.random.default_rng(5)
    settings = [_settings(random_inside_view(rng, *((200, 120), (64, 48))[i % 2]), deg=0) for i in range(16)]
    br = BatchedRasterizer(settings, g)
    br.forward()
    torch.cuda.synchronize()
    br.status()
    for v, rs in enumerate(settings):
        img = dmgs_gb300.GaussianRasterizer(rs)(means2D=torch.zeros_like(g["means3D"]), **g)[0]
        assert torch.equal(br.images[v], img), v
