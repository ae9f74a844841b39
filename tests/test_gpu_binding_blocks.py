"""The bindings at the edges of their blocks (64 faces each, fewer where their rows do not fit), with more
Gaussians per face than a block has threads, at odd addresses and with faces
whose indices are out of range, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from dmgs_gb300.binding import bind_faces, bind_faces_scale_rot
from helpers import rel_l2
from oracle import binding as OB

pytestmark = pytest.mark.gpu
D = "cuda"


def _at(a, off):
    """The array on the device, `off` floats past an aligned address."""
    a = np.ascontiguousarray(a, np.float32)
    buf = torch.zeros(a.size + off, device=D)
    t = buf[off:].view(a.shape)
    t.copy_(torch.tensor(a))
    return t


def _mesh(F, seed):
    rng = np.random.default_rng(seed)
    V = max(3, F // 2 + 3)
    faces = np.stack([rng.permutation(V)[:3] for _ in range(F)])
    return rng, rng.standard_normal((V, 3)), faces


CASES = [(1, 1), (1, 64), (1, 65), (3, 64), (3, 65), (6, 63), (6, 65), (7, 100), (127, 3), (300, 3), (700, 2), (1300, 2)]


@pytest.mark.parametrize("G,F", CASES)
@pytest.mark.parametrize("off", [0, 1])
def test_stage2(G, F, off):
    rng, v, f = _mesh(F, G + F)
    bc = rng.dirichlet((1, 1, 1), G)
    gx, gc = rng.standard_normal((F * G, 3)), rng.standard_normal((F * G, 6))
    verts, sf = _at(v, off).requires_grad_(True), torch.tensor([0.3], device=D, requires_grad=True)
    xyz, cov, _ = bind_faces(verts, torch.tensor(f, device=D), _at(bc, off), sf, 0.2, 1.0)
    g = torch.autograd.grad([xyz, cov], [verts, sf], [_at(gx, off), _at(gc, off)])
    v64 = torch.tensor(v.astype(np.float32)).double().requires_grad_(True)
    s64 = torch.tensor([0.3], dtype=torch.float32).double().requires_grad_(True)
    b64 = torch.tensor(bc.astype(np.float32)).double()
    rx, rc, _, _ = OB.bind_stage2(v64, torch.tensor(f), b64, 0.2, 1e-6, s64)
    r = torch.autograd.grad([rx, rc], [v64, s64], [torch.tensor(gx), torch.tensor(gc)])
    for a, b in ((xyz, rx), (cov, rc), (g[0], r[0])):
        assert rel_l2(a.detach().cpu().numpy(), b.detach().numpy()) <= 1e-5
    assert abs(float(g[1]) - float(r[1])) <= 1e-4 * (abs(float(r[1])) + float(rc.detach().abs().sum()))


@pytest.mark.parametrize("G,F", CASES)
@pytest.mark.parametrize("off", [0, 1])
def test_stage3(G, F, off):
    rng, v, f = _mesh(F, 7 * G + F)
    bc = rng.dirichlet((1, 1, 1), G)
    s2, r2 = 0.3 * rng.standard_normal((F * G, 2)), rng.standard_normal((F * G, 2))
    gs = [rng.standard_normal((F * G, k)) for k in (3, 3, 4)]
    ins = [_at(a, off).requires_grad_(True) for a in (v, s2, r2)]
    outs = bind_faces_scale_rot(ins[0], torch.tensor(f, device=D), _at(bc, off), ins[1], ins[2], 1e-4)
    g = torch.autograd.grad(outs, ins, [_at(a, off) for a in gs])
    i64 = [torch.tensor(a.astype(np.float32)).double().requires_grad_(True) for a in (v, s2, r2)]
    rx, rs, _, rq = OB.bind_stage3(i64[0], torch.tensor(f), torch.tensor(bc.astype(np.float32)).double(), i64[1], i64[2], 1e-4)
    r = torch.autograd.grad([rx, rs, rq], i64, [torch.tensor(a) for a in gs])
    for a, b in zip(outs, (rx, rs, rq)):
        assert rel_l2(a.detach().cpu().numpy(), b.detach().numpy()) <= 1e-5
    for a, b in zip(g, r):
        # the quaternion's Jacobian grows near its branch changes: float32 of
        # up to ~1e2 amplification
        assert rel_l2(a.cpu().numpy(), b.numpy()) <= 1e-4


@pytest.mark.parametrize("G", [6, 300])
def test_out_of_range_faces_are_skipped(G):
    rng, v, f = _mesh(60, 5)
    bad = f.copy()
    bad[[0, 17, 59], [0, 1, 2]] = [-1, 10**6, 2**40]
    keep = np.setdiff1d(np.arange(60), [0, 17, 59])
    bc = rng.dirichlet((1, 1, 1), G)
    s2, r2 = rng.standard_normal((60 * G, 2)), rng.standard_normal((60 * G, 2))
    gs = [rng.standard_normal((60, G, k)) for k in (3, 6, 3, 4)]

    def run(faces, rows):
        n = len(rows) * G
        verts = _at(v, 0).requires_grad_(True)
        t = lambda a: _at(a.reshape(60, G, -1)[rows].reshape(n, -1), 0)  # noqa: E731
        fd = torch.tensor(np.ascontiguousarray(faces[rows]), device=D)
        x2, c2, _ = bind_faces(verts, fd, _at(bc, 0), None, 0.2, 1.0)
        (d2,) = torch.autograd.grad([x2, c2], [verts], [t(gs[0]), t(gs[1])])
        x3 = bind_faces_scale_rot(verts, fd, _at(bc, 0), t(s2), t(r2), 1e-4)
        (d3,) = torch.autograd.grad(x3, [verts], [t(gs[0]), t(gs[2]), t(gs[3])])
        return [x2, c2, *x3], [d2, d3]
    a, da = run(bad, np.arange(60))
    b, db = run(f, keep)
    for x, y in zip(a, b):
        assert torch.equal(x.view(60, G, -1)[torch.tensor(keep, device=D)], y.view(57, G, -1))
    for x, y in zip(da, db):
        assert rel_l2(x.cpu().numpy(), y.cpu().numpy()) <= 1e-5
