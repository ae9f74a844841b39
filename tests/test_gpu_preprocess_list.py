"""The single-view preprocess's list of visible Gaussians (colours evaluated by
the block's first threads) against the batched form's, bit for bit, at the
edges of warps and blocks and with none, some and all visible."""
import pytest
import torch

import dmgs_gb300
from dmgs_gb300.batched import BatchedRasterizer
from test_gpu_batched import D, _scene_and_views, _settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 31, 33, 255, 256, 257, 513])
@pytest.mark.parametrize("visible", ["none", "every 5th", "all"])
def test_colours_of_listed_gaussians(P, visible):
    _, views = _scene_and_views(P=8, seed=3)
    rs = _settings(views[1], bg=(0.1, 0.2, 0.3))
    gen = torch.Generator(device=D).manual_seed(P)
    g = {"means3D": torch.rand(P, 3, device=D, generator=gen) - 0.5,
         "opacities": 0.2 + 0.7 * torch.rand(P, 1, device=D, generator=gen),
         "shs": torch.randn(P, 16, 3, device=D, generator=gen),
         "scales": 0.02 + 0.1 * torch.rand(P, 3, device=D, generator=gen),
         "rotations": torch.nn.functional.normalize(torch.randn(P, 4, device=D, generator=gen))}
    hide = torch.ones(P, dtype=torch.bool, device=D)
    if visible != "none":
        hide[::5 if visible == "every 5th" else 1] = False
    g["means3D"][hide] += 3 * rs.campos  # behind the camera, which looks at the origin
    img, radii = dmgs_gb300.GaussianRasterizer(rs)(means2D=torch.zeros_like(g["means3D"]), **g)
    assert torch.equal(radii > 0, ~hide)
    br = BatchedRasterizer([rs, rs], g)
    br.forward()
    torch.cuda.synchronize()
    br.status()
    for v in range(2):
        assert torch.equal(br.images[v], img)
        assert torch.equal(br.radii[v], radii)
