"""The texture's MLP tiles of 128 points: ragged last tiles, several tiles a
block, and the forward without a kept encoding, per channel count."""
import pytest
import torch

from dmgs_gb300.texture import MLPTexture3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [3, 12, 27, 48])
@pytest.mark.parametrize("n", [1, 63, 65, 127, 128, 129, 152 * 4 * 128 + 1])
def test_mlp_tiles_match_float64(channels, n):
    g = torch.Generator().manual_seed(1000 * channels + n)
    tex = MLPTexture3D(torch.tensor([[-1.0] * 3, [1.0] * 3]), channels=channels, device="cuda")
    ws = [w for w in tex.net.weights()]
    with torch.no_grad():
        tex.encoder.params.copy_(torch.randn(tex.encoder.params.shape, generator=g))
        for w in ws:
            w.copy_(0.3 * torch.randn(w.shape, generator=g))
    x = (2.2 * torch.rand(n, 3, generator=g) - 1.1).cuda()
    d = torch.randn(n, channels, generator=g).cuda()
    out = tex.sample_noact(x)
    with torch.no_grad():  # no encoding kept: the same kernel, the same bits
        assert torch.equal(tex.sample_noact(x), out)
    got = torch.autograd.grad(out, ws, d)

    # the encoding by itself: an MLP of identities (up to its ReLU) reads it out
    def encoding():
        parts = []
        for sign in (1.0, -1.0):
            probe = MLPTexture3D(torch.tensor([[-1.0] * 3, [1.0] * 3]), channels=48, device="cuda")
            with torch.no_grad():
                probe.encoder.params.copy_(tex.encoder.params)
                for w, v in zip(probe.net.weights(), (sign * torch.eye(32), torch.eye(32), torch.eye(48, 32))):
                    w.copy_(v)
                parts.append(sign * probe.sample_noact(x)[:, :32])
        return (parts[0] + parts[1]).double()
    w64 = [w.detach().double().requires_grad_(True) for w in ws]
    h = encoding()
    for w in w64[:2]:
        h = torch.relu(h @ w.T)
    ref = h @ w64[2].T
    # three float32 layers of 32 terms each: 96 roundings of 2^-24 against the norm
    assert float((out.detach().double() - ref.detach()).norm()) <= 96 * 2 ** -24 * float(ref.detach().norm())
    for a, b in zip(got, torch.autograd.grad(ref, w64, d.double())):
        # a float32 sum over n points of terms of either sign, and units whose sign a rounding flips
        assert float((a.double() - b).norm()) <= 1e-4 * float(b.norm())
