"""Twenty views of one scene in one batch, on fresh contexts again and again: every launch gives the same bits.
Sorts that run side by side leave every view's digit histograms in other caches at the time its passes start,
so a pass that read them before waiting for the kernel in front of it now and then saw an unfinished one."""
import numpy as np
import pytest

import webgs
from webgs import workloads as W

pytestmark = pytest.mark.gpu


def test_batches_repeat_bit_for_bit():
    spec = W.SceneSpec(60_000, 4, 1, 64, 20.0)
    packed = spec.build()
    views = [c.view() for _, c in W.orbit_cameras(20, 17, 9.0, resolutions=((96, 64), (128, 96)))]
    first = None
    for _ in range(40):
        with webgs.Context() as ctx:
            sc = ctx.upload(packed, spec.count)
            out = [o["rgba8"] for o in ctx.forward_batch([(sc, v) for v in views])]
            sc.close()
        if first is None:
            first = out
        for a, b in zip(first, out):
            np.testing.assert_array_equal(a, b)
