"""The emit's largest partitions (2048 Gaussians, from 8 million up): one frame of a little over 8 million Gaussians
through the properties of test_gpu_full_size.py, with a budget that holds all instances and one that cuts them off."""
import numpy as np
import pytest

import webgs
from test_gpu_full_size import _check
from webgs import workloads as W

pytestmark = pytest.mark.gpu
N = 8_000_000 + 1027  # the last partition is a partial one


@pytest.fixture(scope="module")
def packed():
    small = 100_000
    base = W.SceneSpec(small, 9, 0).build()
    out = np.empty(59 * N, np.float32)
    at = 0
    for width in (3, 3, 4, 3, 1, 45):  # the attribute blocks
        out[at * N:(at + width) * N] = np.resize(base[at * small:(at + width) * small], width * N)
        at += width
    out[3 * N:6 * N] -= 2.0
    out[:3 * N] += np.random.default_rng(1).normal(0.0, 0.05, 3 * N).astype(np.float32)
    return out


def test_partitions_of_2048(packed):
    view = W.CameraSpec((0.0, 0.1, -4.0), (0.0, 0.0, 0.0), 60.0, 250, 130).view()
    with webgs.Context(max_instance_factor=4) as ctx:
        sc = ctx.upload(packed, N)
        _check(ctx, sc, view, 250, 130)
        full = ctx.debug()
        sc.close()
    assert full["instance_count"] == full["sorted_count"] > 0
    with webgs.Context(max_instance_factor=1, tile_size=8) as ctx:
        sc = ctx.upload(packed, N)
        out = ctx.forward(sc, view, allow_overflow=True)
        d = ctx.debug()
        sc.close()
    assert "overflow" in out and d["sorted_count"] == N < d["instance_count"]
    assert np.all(np.diff(d["keys"].astype(np.int64)) >= 0)
    kept = np.clip(N - d["offsets"][:-1].astype(np.int64), 0, d["tiles_touched"])
    np.testing.assert_array_equal(np.bincount(d["vals"], minlength=N), kept)
