"""The fused loss at the edges of its small (32 x 16) tiles, and of its large
(32 x 54) ones in images that take those, against the float64 composition; its
scratch follows the tile."""
import pytest
import torch

from dmgs_gb300 import _lib
from dmgs_gb300.loss import l1_ssim_loss
from dmgs_gb300.meshbound import ssim

pytestmark = pytest.mark.gpu


# images of fewer than 304 large tiles take small ones (303 and 304 channels of one large tile each are the rule's two sides)
@pytest.mark.parametrize("C,H,W", [(1, 15, 31), (1, 16, 32), (1, 17, 33), (3, 32, 64), (2, 33, 95), (3, 200, 200), (3, 107, 1727),
                                   (3, 108, 1728), (3, 109, 1729), (303, 20, 30), (304, 20, 30), (304, 55, 33)])
def test_tiles_match_float64(C, H, W):
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W)
    x = torch.rand(C, H, W, device="cuda", generator=g).requires_grad_(True)
    y = (x.detach() + 0.1 * torch.randn(C, H, W, device="cuda", generator=g)).clamp(0, 1)
    loss = l1_ssim_loss(x, y, 0.2)
    loss.backward()
    xd = x.detach().double().requires_grad_(True)
    ref = 0.8 * (xd - y.double()).abs().mean() + 0.2 * (1.0 - ssim(xd, y.double()))
    ref.backward()
    assert abs(float(loss.detach()) - float(ref.detach())) <= 1e-5 * abs(float(ref.detach())) + 1e-7
    d = (x.grad.double() - xd.grad).norm() / xd.grad.norm()
    assert float(d) <= 1e-4


@pytest.mark.parametrize("C,H,W", [(3, 200, 200), (303, 20, 30), (304, 20, 30)])
def test_scratch_is_what_the_call_asks_for(C, H, W):
    """The call writes no byte past dmgs_l1_ssim_scratch_bytes and refuses less."""
    lib = _lib.load()
    n = lib.dmgs_l1_ssim_scratch_bytes(C, H, W)
    x, y = torch.rand(C, H, W, device="cuda"), torch.rand(C, H, W, device="cuda")
    grad, loss = torch.empty_like(x), torch.empty((), device="cuda")
    scratch = torch.full((n + 4096,), 77, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    args = (x.data_ptr(), y.data_ptr(), C, H, W, 0.2, loss.data_ptr(), grad.data_ptr(), scratch.data_ptr())
    assert lib.dmgs_l1_ssim(*args, n - 1, s) == -3
    assert lib.dmgs_l1_ssim(*args, n, s) == 0
    torch.cuda.synchronize()
    assert torch.equal(scratch[n:], torch.full_like(scratch[n:], 77))
