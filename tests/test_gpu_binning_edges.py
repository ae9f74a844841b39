"""The binning's tiles and groups at their edges, and the single-view adjoint's
outputs at odd shapes and addresses."""
import numpy as np
import pytest
import torch

from dmgs_gb300 import _lib
from dmgs_gb300._lib import DmgsGrads
from dmgs_gb300.scenes import small_scene
from helpers import AbiRun, _dev, mode_inputs, rel_l2

pytestmark = pytest.mark.gpu


def _expected_lists(dv, gx, T):
    """Tile lists in (depth, index) order from the per-Gaussian rectangles."""
    ids, tiles = [], []
    vis = np.nonzero(dv["tiles_touched"])[0]
    order = vis[np.lexsort((vis, dv["depth"][vis].view(np.uint32)))]
    for i in order:
        x0, y0, x1, y1 = dv["rect"][i]
        t = (np.arange(y0, y1)[:, None] * gx + np.arange(x0, x1)[None, :]).reshape(-1)
        tiles.append(t)
        ids.append(np.full(t.size, i))
    ids = np.concatenate(ids) if ids else np.zeros(0, np.int64)
    tiles = np.concatenate(tiles) if tiles else np.zeros(0, np.int64)
    o = np.argsort(tiles, kind="stable")
    counts = np.bincount(tiles, minlength=T)
    ends = np.cumsum(counts)
    ranges = np.stack([ends - counts, ends], 1)
    ranges[counts == 0] = 0
    return ids[o], ranges


# 2048 Gaussians per compaction / sort tile, 32 tiles per group of counts
@pytest.mark.parametrize("P", [1, 255, 257, 2047, 2048, 2049, 4097, 65536, 65537, 133_121])
@pytest.mark.parametrize("culled", [0.0, 0.9, 1.0])
def test_lists_at_tile_and_group_edges(P, culled):
    sc = small_scene(P=P, width=100, height=70, seed=P)
    inp = mode_inputs(sc, ("colors", "sr"))
    rng = np.random.default_rng(P + 1)
    m = inp["means3D"].copy()
    m[rng.uniform(size=P) < culled] += np.float32(100.0) * np.asarray([0.47, 0.34, 0.81], np.float32)  # behind the camera
    m[P // 2:] = np.where(rng.uniform(size=(P - P // 2, 1)) < 0.3, m[: P - P // 2], m[P // 2:])  # exact depth ties
    inp["means3D"] = m
    inp["scales"] = inp["scales"] * np.float32((1e3 / max(P, 1000)) ** (1 / 3))
    run = AbiRun(sc.views[0], inp).forward()
    dv = run.debug_views()
    ids, ranges = _expected_lists(dv, 7, 7 * 5)
    assert run.K == ids.size
    np.testing.assert_array_equal(dv["values"], ids)
    np.testing.assert_array_equal(dv["ranges"], ranges)
    if culled == 1.0:
        assert run.K == 0


@pytest.mark.parametrize("M,deg", [(1, 0), (4, 1), (5, 1), (9, 2), (16, 3), (17, 3)])
@pytest.mark.parametrize("off", [0, 1])
def test_adjoint_rows_at_odd_widths_and_addresses(M, deg, off):
    """Every output row written, zero for culled Gaussians, at output
    addresses off by one float (the rotations stay 16-byte aligned): against
    the FP64-sum mode at aligned addresses, whose sums differ by float32
    rounding only."""
    sc = small_scene(P=3000, width=90, height=70, seed=M)
    inp = mode_inputs(sc, ("shs", "sr"))
    inp["means3D"] = inp["means3D"] * np.float32(3.0)  # a good part outside the view
    sh = np.zeros((3000, M, 3), np.float32)
    n = min(M, 16)
    sh[:, :n] = inp["shs"][:, :n]
    inp["shs"] = sh
    run = AbiRun(sc.views[0], inp, sh_degree=deg).forward()
    dimg = np.random.default_rng(1).standard_normal((3, 70, 90)).astype(np.float32)
    ref = run.backward(dimg, f64sum=True)
    P = run.P
    shapes = dict(means2D=(P, 3), opacities=(P, 1), means3D=(P, 3), shs=(P, M, 3), scales=(P, 3), rotations=(P, 4))
    buf = {k: torch.full((int(np.prod(s)) + 8,), float("nan"), device="cuda") for k, s in shapes.items()}
    o = {k: 0 if k == "rotations" else off for k in shapes}
    at = lambda k: buf[k].data_ptr() + 4 * o[k]  # noqa: E731
    grads = DmgsGrads(at("means2D"), None, at("opacities"), at("means3D"), None, at("shs"), at("scales"), at("rotations"))
    scratch = torch.full((run.lib.dmgs_bwd_scratch_bytes(P) // 4,), float("nan"), device="cuda")
    dout = _dev(dimg)
    _lib.check(run.lib.dmgs_raster_bwd(run.view, run.g, dout.data_ptr(), run.geom.data_ptr(), run.geom.numel(),
                                       run.bin.data_ptr(), run.bin.numel(), run.K, run.img.data_ptr(), run.img.numel(),
                                       scratch.data_ptr(), 4 * scratch.numel(), grads, run.stream), "raster_bwd")
    torch.cuda.synchronize()
    vis = run.radii.cpu().numpy() > 0
    assert 0 < vis.sum() < P
    for k, s in shapes.items():
        n = int(np.prod(s))
        b = buf[k].cpu().numpy()
        got = b[o[k]: o[k] + n].reshape(s)
        assert np.isnan(b[: o[k]]).all() and np.isnan(b[o[k] + n:]).all(), k  # nothing beside the array
        assert np.isfinite(got).all() and not got[~vis].any(), k
        assert rel_l2(got, ref[k]) <= 1e-4, k  # float32 sums of ~1e3 terms, amplified by the covariance chain
