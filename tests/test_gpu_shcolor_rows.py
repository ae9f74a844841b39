"""The fused colours at block edges, in the staged form (every coefficient
active) and the per-thread form (more coefficients than the degree needs, or
rows off 16 bytes), against the float64 composition."""
import pytest
import torch

from dmgs_gb300.meshbound import eval_sh
from dmgs_gb300.shcolor import sh_colors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("deg,K", [(0, 1), (1, 4), (2, 9), (3, 16), (1, 16), (2, 11)])
@pytest.mark.parametrize("off", [0, 1])
def test_rows(P, deg, K, off):
    g = torch.Generator(device="cuda").manual_seed(P + 100 * deg)
    buf = 0.4 * torch.randn(P * 3 * K + off, device="cuda", generator=g)
    sh = buf[off:].view(P, 3, K).requires_grad_(True)
    xyz = torch.randn(P, 3, device="cuda", generator=g).requires_grad_(True)
    cam = torch.tensor([0.3, -4.0, 1.0], device="cuda")
    dcol = torch.randn(P, 3, device="cuda", generator=g)
    col = sh_colors(deg, sh, xyz, cam)
    dsh, dx = torch.autograd.grad(col, [sh, xyz], dcol)
    s64, x64 = sh.detach().double().requires_grad_(True), xyz.detach().double().requires_grad_(True)
    d = x64 - cam.double()
    ref = torch.sigmoid(eval_sh(deg, s64, d / d.norm(dim=1, keepdim=True)))
    rsh, rx = torch.autograd.grad(ref, [s64, x64], dcol.double(), allow_unused=True)
    rx = torch.zeros_like(x64) if rx is None else rx
    assert (col.double() - ref).abs().max() <= 2e-6
    for a, b in ((dsh, rsh), (dx, rx)):  # float32 sums of at most 16 terms
        assert (a.double() - b).norm() <= 5e-6 * b.norm() + 1e-12
