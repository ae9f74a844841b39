"""The stage-3 binding where several threads share a face's Gaussians (the
faces whose rows fit a block leave threads over), and with one Gaussian per
face, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from dmgs_gb300.binding import bind_faces_scale_rot
from helpers import rel_l2
from oracle import binding as OB
from test_gpu_binding_blocks import D, _at, _mesh

pytestmark = pytest.mark.gpu


# 402 Gaussians' rows fit a block: faces per block, and threads per face, at 12 | 13 | 25 | 26 | 51 | ... per face
@pytest.mark.parametrize("G,F", [(12, 70), (13, 61), (25, 33), (26, 31), (50, 17), (51, 15), (100, 9), (101, 7), (201, 5), (202, 3),
                                 (402, 2), (403, 3), (1000, 2), (1, 1), (1, 257), (2, 130), (3, 65), (3, 128), (4, 63)])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("bad", [False, True])
def test_stage3_at_every_share(G, F, off, bad):
    rng, v, f = _mesh(F, 3 * G + F)
    bc = rng.dirichlet((1, 1, 1), G)
    s2, r2 = 0.3 * rng.standard_normal((F * G, 2)), rng.standard_normal((F * G, 2))
    gs = [rng.standard_normal((F * G, k)) for k in (3, 3, 4)]
    faces = f.copy()
    keep = np.ones(F, bool)
    if bad:  # one face out of range: skipped, and its block's other faces written one by one
        faces[F // 2, 1] = -1
        keep[F // 2] = False
    rows = np.repeat(keep, G)
    ins = [_at(a, off).requires_grad_(True) for a in (v, s2, r2)]
    outs = bind_faces_scale_rot(ins[0], torch.tensor(faces, device=D), _at(bc, off), ins[1], ins[2], 1e-4)
    g = torch.autograd.grad(outs, ins, [_at(a, off) for a in gs])
    if not keep.any():
        assert float(g[0].abs().max()) == 0.0
        return
    i64 = [torch.tensor(a.astype(np.float32)).double().requires_grad_(True) for a in (v, s2[rows], r2[rows])]
    rx, rs, _, rq = OB.bind_stage3(i64[0], torch.tensor(f[keep]), torch.tensor(bc.astype(np.float32)).double(), i64[1], i64[2], 1e-4)
    r = torch.autograd.grad([rx, rs, rq], i64, [torch.tensor(a[rows]) for a in gs])
    sel = torch.tensor(rows, device=D)
    for a, b in zip(outs, (rx, rs, rq)):
        assert rel_l2(a[sel].detach().cpu().numpy(), b.detach().numpy()) <= 1e-5
    for a, b in zip((g[0], g[1][sel], g[2][sel]), r):
        # the quaternion's Jacobian grows near its branch changes: float32 of
        # up to ~1e2 amplification
        assert rel_l2(a.cpu().numpy(), b.numpy()) <= 1e-4
