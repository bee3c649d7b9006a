"""The batched preprocess backward at Gaussian counts on both sides of a CTA's 128 and view counts on both
sides of a group's 16 (and of the 8 whose blocks leave room for a fourth CTA), with Gaussians that some views,
or none, see: each block of attributes against the sum of the views' own gradients in 64 bits.

Tolerance: every gradient is a sum of a view's terms rounded to 24 bits; the two orders of adding at most 17 views,
and the chain rule taken after the sum instead of before it, differ by some tens of roundings, 1e-5 of the
block's norm."""
import numpy as np
import pytest

import webgs
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,views", [(1, 2), (127, 9), (128, 16), (129, 8), (1000, 17), (257, 1)])
def test_views_sum(n, views):
    packed = W.SceneSpec(n, 40 + n, 0).build()
    packed[3 * n:6 * n] += 1.5
    packed[:3] = (0.0, 0.0, 300.0)  # seen by no view
    cams = [W.CameraSpec((np.sin(k), 0.1, -4.0 + 0.2 * k), (0.3 * np.cos(k), 0.0, 0.0), 35.0, 61, 45).view() for k in range(views)]
    rng = np.random.default_rng(n)
    dls = [rng.normal(0, 1e-3, (45, 61, 3)).astype(np.float32) for _ in cams]
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE) as ctx:
        sc = ctx.upload(packed, n)
        for _ in range(2):  # the second call starts from the gradients the first one cleared
            ctx.forward_batch([(sc, v) for v in cams], rgba8=False, rgb=True)
            got = ctx.backward_batch(sc, dls).astype(np.float64)
        want = np.zeros(59 * n)
        for v, dl in zip(cams, dls):
            ctx.forward(sc, v, rgba8=False)
            want += ctx.backward(sc, dl)
        sc.close()
    at = 0
    for width in (3, 3, 4, 3, 1, 45):
        a, b = got[at * n:(at + width) * n], want[at * n:(at + width) * n]
        at += width
        assert np.linalg.norm(a - b) <= 1e-5 * max(np.linalg.norm(b), 1e-12), (width, at)
    assert n == 1 or np.abs(want).max() > 0
