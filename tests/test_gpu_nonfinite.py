"""Values that are not finite stay where they arise: what does not depend on
them keeps its value."""
import math

import pytest
import torch

import dmgs_gb300
from dmgs_gb300.binding import barycentric_table, bind_faces_scale_rot

pytestmark = pytest.mark.gpu
D = "cuda"


def _gen(seed):
    return torch.Generator(device=D).manual_seed(seed)


def _bind3(r2, drots):
    v = torch.randn(40, 3, device=D, generator=_gen(1)).requires_grad_(True)
    f = torch.stack([torch.randperm(40, device=D, generator=_gen(2 + i))[:3] for i in range(30)])
    bc, _ = barycentric_table(3, D)
    s2 = 0.1 * torch.randn(90, 2, device=D, generator=_gen(50))
    r2 = r2.clone().requires_grad_(True)
    _, _, q = bind_faces_scale_rot(v, f, bc, s2, r2, 1e-5)
    return (q.detach(), *torch.autograd.grad(q, [v, r2], drots))


@pytest.mark.parametrize("big", [1e19, 2e19, 1e30])
def test_2d_rotation_whose_square_overflows(big):
    """|r|^2 beyond float32's range: r / |r| is 0 there (r / infinity), as for
    a zero row, and the row's own gradient is 0."""
    drots = torch.randn(90, 4, device=D, generator=_gen(60))
    r2 = torch.randn(90, 2, device=D, generator=_gen(61))
    r2[17] = 0.0
    want = _bind3(r2, drots)
    r2[17] = torch.tensor([big, -0.5 * big])
    got = _bind3(r2, drots)
    if big * big * 1.25 < 3.4e38:  # the square still fits: a plain rotation
        want = _bind3(torch.where(torch.arange(90, device=D)[:, None] == 17, r2 / big, r2), drots)
        assert torch.allclose(got[0], want[0], rtol=1e-5, atol=1e-6)
        return
    assert all(bool(torch.isfinite(t).all()) for t in got)
    assert torch.equal(got[0], want[0])
    assert torch.equal(got[2][17], torch.zeros(2, device=D))
    keep = torch.arange(90, device=D) != 17
    assert torch.equal(got[2][keep], want[2][keep])


def _pixel_settings(w, h):
    """A camera at the origin looking along +z: the point (x, y, z) of pixel (i, j)
    at depth 1 is ((2 i + 1) / w - 1, (2 j + 1) / h - 1, 1)."""
    n, f = 0.01, 100.0
    proj = torch.zeros(4, 4, device=D)
    proj[0, 0] = proj[1, 1] = 1.0
    proj[2, 2], proj[2, 3], proj[3, 2] = f / (f - n), -f * n / (f - n), 1.0
    return dmgs_gb300.GaussianRasterizationSettings(
        image_height=h, image_width=w, tanfovx=1.0, tanfovy=1.0, bg=torch.tensor([0.2, 0.3, 0.4], device=D), scale_modifier=1.0,
        viewmatrix=torch.eye(4, device=D), projmatrix=proj.T.contiguous(), sh_degree=0, campos=torch.zeros(3, device=D),
        prefiltered=False, debug=False)


@pytest.mark.parametrize("others", [0, 40_000])  # a short work list's strips, a long one's halves
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3e38])
@pytest.mark.parametrize("channels", [(0, 1, 2), (0,), (2,)])
def test_pixel_gradient_that_is_not_finite_stays_with_its_gaussians(others, bad, channels):
    """Two Gaussians a warp visits together, one of them at a pixel whose
    gradient is not finite: the other one's mean, covariance and opacity
    gradients are those without that pixel."""
    w = h = 256
    rs = _pixel_settings(w, h)
    g = _gen(7)
    px = torch.tensor([[3.0, 1.0], [12.0, 1.0]], device=D)
    if others:
        px = torch.cat([px, 32 + 220 * torch.rand(others, 2, device=D, generator=g)])
    P = px.shape[0]
    means = torch.cat([(2 * px + 1) / w - 1, torch.ones(P, 1, device=D)], 1)
    t_color = 1.0 + 4.0 * torch.rand(P, 3, device=D, generator=g)  # above 1: the largest finite gradient overflows
    means[:, 2] += 0.001 * torch.rand(P, device=D, generator=g)
    sigma = 0.6 * 2 / w
    cov = torch.tensor([sigma ** 2, 0, 0, sigma ** 2, 0, sigma ** 2], device=D).repeat(P, 1)
    t = dict(means3D=means, opacities=torch.full((P, 1), 0.1 if others else 0.8, device=D), colors_precomp=t_color,
             cov3D_precomp=cov, means2D=torch.zeros(P, 3, device=D))
    t["opacities"][:2] = 0.8
    for x in t.values():
        x.requires_grad_(True)
    dimg = torch.randn(3, h, w, device=D, generator=g)

    def grads(value):
        d = dimg.clone()
        d[list(channels), 1, 3] = value
        img, radii = dmgs_gb300.GaussianRasterizer(rs)(**t)
        assert int(radii[:2].min()) > 0
        return dict(zip(t, torch.autograd.grad(img, list(t.values()), d)))
    want, got = grads(0.0), grads(bad)
    for k in ("means3D", "opacities", "cov3D_precomp", "means2D"):
        assert bool(torch.isfinite(want[k][1]).all()) and float(want[k][1].abs().max()) > 0
        if bad != 3e38:
            assert not bool(torch.isfinite(got[k][0]).all())  # the Gaussian of the pixel itself
        # one Gaussian, few pixels: the same terms, added a strip or a half of
        # a tile at a time (rounding, with terms up to a thousand times the sum)
        assert torch.allclose(got[k][1], want[k][1], rtol=1e-4, atol=0), k


def test_loss_gradient_where_a_square_overflows():
    """A pixel whose square overflows: E[x^2] is infinite in its window, SSIM
    and its derivatives 0 there, and every gradient stays finite."""
    from dmgs_gb300.loss import l1_ssim_loss
    x = torch.rand(1, 40, 40, device=D, generator=_gen(70))
    y = torch.rand(1, 40, 40, device=D, generator=_gen(71))
    x[0, 20, 20] = 2.5e19
    x.requires_grad_(True)
    (g,) = torch.autograd.grad(l1_ssim_loss(x, y, 0.2), [x])
    assert bool(torch.isfinite(g).all())
    # in the pixel's own window only the L1 term is left
    assert math.isclose(float(g[0, 20, 20]), 0.8 / 1600, rel_tol=1e-5)
