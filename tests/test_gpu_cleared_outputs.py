"""The outputs that the blend adjoint clears, from one item of work to many:
every element written (they start as NaN), zero where a Gaussian is culled, and
the FP64-sum mode's gradients where it is not."""
import numpy as np
import pytest

from dmgs_gb300.scenes import small_scene
from helpers import AbiRun, mode_inputs, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,w,h", [(1, 16, 16), (50, 16, 16), (5000, 16, 16), (70_001, 16, 16), (70_001, 33, 17), (70_001, 300, 200),
                                   (400_000, 16, 16), (400_000, 100, 100)])
@pytest.mark.parametrize("culled", [0.5, 1.0])
def test_every_output_is_written(P, w, h, culled):
    sc = small_scene(P=P, width=w, height=h, seed=P % 1000)
    inp = mode_inputs(sc, ("shs", "sr"))
    rng = np.random.default_rng(P)
    m = inp["means3D"].copy()
    away = rng.uniform(size=P) < culled
    m[away] += np.float32(100.0) * np.asarray([0.47, 0.34, 0.81], np.float32)  # behind the camera
    inp["means3D"] = m
    inp["scales"] = inp["scales"] * np.float32((1e3 / max(P, 1000)) ** (1 / 3))
    run = AbiRun(sc.views[0], inp).forward()
    dout = rng.standard_normal((3, h, w)).astype(np.float32)
    got, want = run.backward(dout), run.backward(dout, f64sum=True)
    hidden = run.radii.cpu().numpy()[:P] <= 0
    assert hidden.sum() >= away.sum()
    for k, a in got.items():
        if a is None:
            continue
        assert np.isfinite(a).all(), k
        assert not a[hidden].any(), k
        if (~hidden).any() and np.abs(want[k]).max() > 0:
            # the sums' order alone: float32 rounding over a Gaussian's pixels,
            # amplified by the covariance chain of needles
            assert rel_l2(a, want[k]) <= 1e-3, k
