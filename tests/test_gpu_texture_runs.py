"""The texture adjoint's table reduction, one per run of consecutive points in
the same cell: the gradients do not depend on the points' order."""
import pytest
import torch

from dmgs_gb300.texture import MLPTexture3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 33, 257, 1000])
@pytest.mark.parametrize("spread", [0.0, 1e-3, 0.05, 1.0])
def test_gradients_do_not_depend_on_the_order_of_the_points(n, spread):
    torch.manual_seed(n)
    tex = MLPTexture3D(torch.tensor([[-1.0] * 3, [1.0] * 3]), channels=12, device="cuda")
    with torch.no_grad():
        tex.encoder.params.copy_(torch.randn_like(tex.encoder.params))
    # a walk: neighbours share cells on some levels, not on others
    step = spread * torch.randn(n, 3, device="cuda") / n
    x = (0.1 + torch.cumsum(step, 0)).clamp(-1.2, 1.2)
    d = torch.randn(n, 12, device="cuda")
    perm = torch.randperm(n, device="cuda")

    def grads(xs, ds):
        xs = xs.clone().requires_grad_(True)
        out = tex.sample_noact(xs)
        return torch.autograd.grad(out, [xs, tex.encoder.params], ds)
    a, b = grads(x, d), grads(x[perm], d[perm])
    assert torch.equal(a[0][perm], b[0])
    # float32 sums of up to n terms per entry in another order
    assert float((a[1].double() - b[1].double()).norm()) <= 2e-5 * float(b[1].double().norm())
    assert int((a[1] != 0).sum()) == int((b[1] != 0).sum())
    # each gradient by itself: the position gradient is not reduced over points
    xs = x.clone().requires_grad_(True)
    tex.encoder.params.requires_grad_(False)
    assert torch.equal(torch.autograd.grad(tex.sample_noact(xs), xs, d)[0], a[0])
    tex.encoder.params.requires_grad_(True)
    t = torch.autograd.grad(tex.sample_noact(x), tex.encoder.params, d)[0]
    assert float((a[1].double() - t.double()).norm()) <= 2e-5 * float(t.double().norm())
