"""Images of more than 512 tiles a row: the emission's row pieces, groups of
Gaussians with none in a piece among them.  Lists against the per-Gaussian
rectangles."""
import numpy as np
import pytest

from helpers import AbiRun
from test_gpu_binning_edges import _expected_lists

pytestmark = pytest.mark.gpu


class _View:
    """A camera at the origin looking along +z; pixel (i, j) at depth 1 is at
    (2 i + 1 - w, 2 j + 1 - h) / w (square pixels)."""

    def __init__(self, w, h):
        n, f = 0.01, 100.0
        self.width, self.height, self.tanfovx, self.tanfovy = w, h, 1.0, h / w
        p = np.zeros((4, 4), np.float32)
        p[0, 0], p[1, 1] = 1.0, w / h
        p[2, 2], p[2, 3], p[3, 2] = f / (f - n), -f * n / (f - n), 1.0
        self.viewmatrix, self.projmatrix = np.eye(4, dtype=np.float32), np.ascontiguousarray(p.T)
        self.campos = np.zeros(3, np.float32)


# 512, 513, 1024 and 1875 tiles a row; 1 and 3 rows
@pytest.mark.parametrize("w,h", [(8192, 16), (8193, 16), (8208, 40), (16384, 16), (30000, 16), (30000, 48)])
@pytest.mark.parametrize("order", ["by place", "shuffled"])
def test_lists_by_row_piece(w, h, order):
    """Gaussians whose depth order follows their place leave every group of 32
    in one stretch of the row."""
    P = 3000
    rng = np.random.default_rng(w + h)
    x = np.sort(rng.uniform(0, w, P))
    y = rng.uniform(0, h, P)
    z = 1.0 + 1e-4 * np.arange(P)
    if order == "shuffled":
        z = rng.permutation(z)
    z = z.astype(np.float32)
    means = np.stack([(2 * x + 1 - w) / w * z, (2 * y + 1 - h) / w * z, z], 1).astype(np.float32)
    sigma = (rng.choice([1.0, 30.0, 400.0], P, p=[0.6, 0.35, 0.05]) * 2 / w).astype(np.float32)
    cov = np.zeros((P, 6), np.float32)
    cov[:, 0], cov[:, 3], cov[:, 5] = sigma ** 2, (2.0 / w) ** 2, (2.0 / w) ** 2
    inp = dict(means3D=means, opacities=np.full((P, 1), 0.3, np.float32), shs=None, colors=rng.uniform(size=(P, 3)).astype(np.float32),
               scales=None, rotations=None, cov3D=cov)
    run = AbiRun(_View(w, h), inp).forward()
    dv = run.debug_views()
    gx, gy = -(-w // 16), -(-h // 16)
    ids, ranges = _expected_lists(dv, gx, gx * gy)
    assert run.K == ids.size > 1000
    np.testing.assert_array_equal(dv["values"], ids)
    np.testing.assert_array_equal(dv["ranges"], ranges)
    grads = run.backward(rng.standard_normal((3, h, w)).astype(np.float32))
    assert all(np.isfinite(g).all() for g in grads.values() if g is not None)
