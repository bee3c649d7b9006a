"""The autotuner times each raster once: depths that come to the same step of the raster (128 and 256; all of them in
8x8 tiles) are one candidate, the largest, so the three that it times again are three different kernels."""
import pytest

import webgs
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,size", [(3_000, (96, 64)), (20_000, (320, 240)), (60_000, (250, 130)), (100_000, (640, 480))])
def test_a_pick_is_the_largest_depth_of_its_step(n, size):
    views = [W.CameraSpec((0.0, 0.2 * k, -4.0), (0, 0, 0), 60.0, *size).view() for k in range(2)]
    cfg, ms = webgs.autotune(W.SceneSpec(n, 7, 0).build(), n, views, iters=2)
    assert ms > 0 and cfg["raster_batch"] in ((256,) if cfg["tile_size"] == 8 else (32, 64, 256)), cfg
