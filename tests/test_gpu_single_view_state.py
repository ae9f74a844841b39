"""The single-view entry points against the buffers they are given: what a call
may write and what it leaves alone."""
import ctypes as C

import numpy as np
import pytest
import torch

from dmgs_gb300 import _lib
from dmgs_gb300._lib import DmgsGrads, DmgsView, ptr
from dmgs_gb300.scenes import small_scene
from helpers import AbiRun, mode_inputs

pytestmark = pytest.mark.gpu
D = "cuda"


@pytest.mark.parametrize("n", [2, 4])
def test_renders_of_one_geometry_at_the_same_time(n):
    """Renders of one geometry state with their own binning and image states,
    each on its own stream and with its own background: each the image of a
    render by itself, and the geometry state as it was."""
    sc = small_scene(P=20_000, width=700, height=500, seed=4)
    run = AbiRun(sc.views[0], mode_inputs(sc, ("colors", "sr")), debug=False).forward()
    lib, W, H = run.lib, run.W, run.H
    bgs = [torch.rand(3, device=D, generator=torch.Generator(device=D).manual_seed(i)) for i in range(n)]
    views = [DmgsView(W, H, run.view.tanfovx, run.view.tanfovy, 1.0, 3, 0, 0, ptr(b), *[ptr(t) for t in run.cam_t[1:]]) for b in bgs]
    z = lambda t: [torch.empty_like(t) for _ in range(n)]  # noqa: E731
    bins, imgs, outs = z(run.bin), z(run.img), z(run.color)

    def render(i, stream):
        _lib.check(lib.dmgs_raster_fwd_render(views[i], run.g, run.geom.data_ptr(), run.geom.numel(), bins[i].data_ptr(),
                                              bins[i].numel(), run.K, imgs[i].data_ptr(), imgs[i].numel(), ptr(outs[i]),
                                              stream.cuda_stream), "fwd_render")
    want = []
    for i in range(n):
        render(i, torch.cuda.current_stream())
        want.append(outs[i].clone())
    assert not torch.equal(want[0], want[1])
    geom = run.geom.clone()
    streams = [torch.cuda.Stream() for _ in range(n)]
    torch.cuda.synchronize()
    for _ in range(20):
        for o in outs:
            o.fill_(-1.0)
        torch.cuda.synchronize()
        for i in range(n):
            render(i, streams[i])
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert torch.equal(o, w)
    assert torch.equal(run.geom, geom)  # nothing written: no error, and no state of a render


def test_refused_adjoint_leaves_its_outputs():
    """More SH coefficients than the single-view adjoint takes: an error before
    anything is enqueued."""
    P, M = 64, 125
    sc = small_scene(P=P, width=40, height=24, seed=2)
    inp = mode_inputs(sc, ("shs", "sr"))
    inp["shs"] = np.concatenate([inp["shs"], np.zeros((P, M - inp["shs"].shape[1], 3), np.float32)], 1)
    run = AbiRun(sc.views[0], inp).forward()
    dout = torch.randn(3, 24, 40, device=D)
    outs = [torch.full((P, n), 7.0, device=D) for n in (3, 1, 3, 3 * M, 3, 4)]
    m2, op, m3, sh, s, r = outs
    gr = DmgsGrads(ptr(m2), None, ptr(op), ptr(m3), None, ptr(sh), ptr(s), ptr(r))
    scratch = torch.empty(run.lib.dmgs_bwd_scratch_bytes(P), dtype=torch.uint8, device=D)
    code = run.lib.dmgs_raster_bwd(run.view, run.g, ptr(dout), run.geom.data_ptr(), run.geom.numel(), run.bin.data_ptr(),
                                   run.bin.numel(), run.K, run.img.data_ptr(), run.img.numel(), scratch.data_ptr(),
                                   scratch.numel(), C.byref(gr), run.stream)
    torch.cuda.synchronize()
    assert code == -1 and b"SH coefficients" in run.lib.dmgs_last_error()
    for t in outs:
        assert torch.equal(t, torch.full_like(t, 7.0))
