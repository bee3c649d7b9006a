"""The raster against the oracle, bit for bit, at list lengths on both sides of what it handles at once
(pairs, 32 hits per chunk, a list of 64, groups of 32 positions, steps of 128 and 512), in every tile
size: faint splats, so that every list is walked to its end, and opaque ones, so that pixels end at
different places of it."""
import numpy as np
import pytest

import webgs
from helpers import assert_frame_parity, gpu_frame, oracle_frame
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("logit", [-3.0, 2.0])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 64, 65, 127, 129, 512, 513, 700, 1100])
def test_list_lengths(n, logit, tile):
    packed = W.SceneSpec(n, 900 + n, 0).build()
    packed[:3 * n] *= 0.3
    packed[3 * n:6 * n] += 3.0  # every splat covers most of the image
    packed[13 * n:14 * n] = logit + 0.3 * packed[13 * n:14 * n]
    view = W.CameraSpec((0.05, 0.1, -4.0), (0.0, 0.0, 0.0), 40.0, 45, 37).view()
    for batch in (32, 256):
        with webgs.Context(tile_size=tile, raster_batch=batch) as ctx:
            sc = ctx.upload(packed, n)
            g = gpu_frame(ctx, sc, view)
            plain = ctx.forward(sc, view)  # without the contributor count and the transmittance
            sc.close()
        assert_frame_parity(g, oracle_frame(view, packed, n, tile=tile))
        np.testing.assert_array_equal(plain["rgba8"], g["rgba8"])
