"""The fused loss at the edges of its 32 x 54 tiles, against the float64
composition."""
import pytest
import torch

from dmgs_gb300.loss import l1_ssim_loss
from dmgs_gb300.meshbound import ssim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 3])
@pytest.mark.parametrize("H,W", [(1, 1), (3, 40), (53, 31), (54, 32), (55, 33), (64, 42), (107, 65), (163, 97)])
def test_tiles_match_float64(C, H, W):
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W)
    x = torch.rand(C, H, W, device="cuda", generator=g).requires_grad_(True)
    y = (x.detach() + 0.1 * torch.randn(C, H, W, device="cuda", generator=g)).clamp(0, 1)
    loss = l1_ssim_loss(x, y, 0.2)
    loss.backward()
    xd = x.detach().double().requires_grad_(True)
    ref = 0.8 * (xd - y.double()).abs().mean() + 0.2 * (1.0 - ssim(xd, y.double()))
    ref.backward()
    assert abs(float(loss) - float(ref)) <= 1e-5 * abs(float(ref)) + 1e-7
    d = (x.grad.double() - xd.grad).norm() / xd.grad.norm()
    assert float(d) <= 1e-4
