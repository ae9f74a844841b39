"""What a view holds between forward and backward (sizes alone: no GPU)."""
import pytest

from dmgs_gb300 import _lib
from dmgs_gb300.build import build


# bytes of the geometry state when a view's sort kept separate digit histograms and no list of visible Gaussians
@pytest.mark.parametrize("P,w,h,most", [(3_000_000, 1237, 822, 221_537_536), (1_000_000, 1237, 822, 74_504_960),
                                        (1_000_000, 800, 800, 74_277_120), (272_000, 800, 800, 20_756_480),
                                        (100_000, 800, 800, 8_112_128), (10_000, 256, 256, 912_128)])
def test_geometry_state_of_ordinary_scenes(P, w, h, most):
    build()
    assert _lib.load().dmgs_geom_state_bytes(P, w, h) <= most


def test_growth_per_gaussian_and_per_tile():
    build()
    size = _lib.load().dmgs_geom_state_bytes
    # 48 record + 1 flag + 4 visible list + 4 + 4 sorted + 8 sort copy / rectangles, 2 look-back words and 1/256
    assert (size(20_480_000, 64, 64) - size(0, 64, 64)) / 20_480_000 < 71.1
    # 128 segment counts + 8 range + 64 lists by class
    tiles = 400 * 300
    assert (size(0, 6400, 4800) - size(0, 6400, 16)) / tiles < 201 + 2048 * 4 / 400
