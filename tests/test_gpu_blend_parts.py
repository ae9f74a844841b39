"""The default blend kernels (a warp per part of a tile) against the
CTA-per-tile form of the tuning configurations: list lengths around the
32-entry batches, images whose tiles are blended as strips (few tiles) and as
halves (many), ragged edges."""
import numpy as np
import pytest
import torch

import dmgs_gb300
from dmgs_gb300.batched import BatchedRasterizer
from dmgs_gb300.camera import make_view
from helpers import rel_l2

pytestmark = pytest.mark.gpu


def _scene(n, width, height, seed):
    """n Gaussians inside every 16 x 16 tile of the image, at distinct depths,
    a third of them reaching into the neighbouring tiles."""
    rng = np.random.default_rng(seed)
    view = make_view((0.0, 0.0, -4.0), (0.0, 0.0, 0.0), width, height, fovx_deg=50.0)
    f = width / (2 * view.tanfovx)
    gx, gy = -(-width // 16), -(-height // 16)
    ty, tx = np.divmod(np.repeat(np.arange(gx * gy), n), gx)
    z = 3.0 + 2.0 * rng.uniform(size=tx.size)
    px = np.minimum(tx * 16 + rng.uniform(1, 15, tx.size), width - 1)
    py = np.minimum(ty * 16 + rng.uniform(1, 15, tx.size), height - 1)
    cam = np.stack([(px - (width - 1) / 2) / f * z, (py - (height - 1) / 2) / f * z, z], 1)
    V = view.viewmatrix.astype(np.float64).T  # world -> view
    means = (cam - V[:3, 3]) @ V[:3, :3]
    P = tx.size
    s = np.where(rng.uniform(size=(P, 1)) < 0.33, 8.0, 1.0) * rng.uniform(0.5, 2.0, (P, 3)) * z[:, None] / f
    q = rng.standard_normal((P, 4))
    t = lambda a: torch.tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    g = dict(means3D=t(means), scales=t(s), rotations=t(q / np.linalg.norm(q, axis=1, keepdims=True)),
             opacities=t(rng.uniform(0.02, 1.0, (P, 1))), colors_precomp=t(rng.uniform(size=(P, 3))))
    rs = dmgs_gb300.GaussianRasterizationSettings(
        image_height=height, image_width=width, tanfovx=view.tanfovx, tanfovy=view.tanfovy, bg=t([0.1, 0.2, 0.3]),
        scale_modifier=1.0, viewmatrix=t(view.viewmatrix), projmatrix=t(view.projmatrix), sh_degree=0,
        campos=t(view.campos), prefiltered=False, debug=False)
    return rs, g


@pytest.mark.parametrize("n", [1, 11, 32, 65])
@pytest.mark.parametrize("width,height", [(41, 23), (709, 699)])
def test_parts_match_the_cta_form(n, width, height):
    rs, g = _scene(n, width, height, 10 * n + width)
    br = BatchedRasterizer([rs], g)
    br.dL_dout[0].normal_(generator=torch.Generator(device="cuda").manual_seed(1))
    br.step()
    br.status()
    image = br.images[0].clone()
    grads = {k: v.clone() for k, v in br.grads.items() if v is not None}
    br.set_config(2, 256, 0)
    br.step()
    assert torch.equal(image, br.images[0])
    assert float(image.std()) > 0.01
    for k, v in grads.items():
        # float32 sums of up to ~10^3 terms in another order
        assert rel_l2(v.cpu().numpy(), br.grads[k].cpu().numpy()) <= 2e-5, k


def test_one_long_list_among_short_ones():
    """2,000 Gaussians on one tile, one on each of the others: the long list
    is split into strips, the rest are not."""
    rs, g = _scene(1, 709, 699, 3)
    rs2, h = _scene(2000, 16, 16, 4)  # the first tile's corner of another camera
    P = g["means3D"].shape[0]
    extra = {k: v.clone() for k, v in h.items()}
    c = g["means3D"][P // 2]
    extra["means3D"] = c + (extra["means3D"] - extra["means3D"].mean(0)) * 0.02
    extra["scales"] = extra["scales"] * 0.02
    extra["opacities"] = extra["opacities"] * 0.05
    g = {k: torch.cat([g[k], extra[k]]) for k in g}
    br = BatchedRasterizer([rs], g)
    br.dL_dout[0].normal_(generator=torch.Generator(device="cuda").manual_seed(2))
    br.step()
    assert br.counters()[0]["maxlist"] > 500
    image = br.images[0].clone()
    br.set_config(4, 256, 0)
    br.forward()
    assert torch.equal(image, br.images[0])
