"""The emit at scene sizes on both sides of its partitions (256 to 2048 Gaussians) and of the sizes where it
changes between them, with and without an instance budget that truncates it, bit for bit against the oracle."""
import pytest

import webgs
from helpers import assert_frame_parity, gpu_frame, oracle_frame
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factor", [64, 1])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 511, 513, 74_999, 75_000, 149_999, 150_001])
def test_partition_sizes(n, factor):
    spec = W.SceneSpec(n, 300 + n % 97, 0)
    packed = spec.build()
    packed[3 * n:6 * n] += 1.0  # several tiles per Gaussian
    view = W.CameraSpec((0.0, 0.1, -4.0), (0.0, 0.0, 0.0), 60.0, 75, 49).view()
    with webgs.Context(tile_size=8, max_instance_factor=factor) as ctx:
        sc = ctx.upload(packed, n)
        out = ctx.forward(sc, view, rgba8=True, rgb=True, final_t=True, n_contrib=True, allow_overflow=True)
        dbg = ctx.debug()
        if "overflow" in out:  # a truncated frame has no outputs here: its intermediates
            assert dbg["instance_count"] > dbg["sorted_count"] == n * factor
            sc.close()
            o = oracle_frame(view, packed, n, tile=8, factor=factor)
            for k in ("offsets", "keys", "vals", "ranges"):
                assert (dbg[k][:len(o[k])] == o[k][:len(dbg[k])]).all(), k
            return
        g = gpu_frame(ctx, sc, view)
        sc.close()
    assert_frame_parity(g, oracle_frame(view, packed, n, tile=8, factor=factor))
