"""Twenty-one small views whose sorts run side by side on the side streams, each in launches of its own: three scenes
of seven views, too few of a scene to share a launch. On fresh contexts again and again every view has the bits of
its single frame. (A sort pass or an emit that read what the kernels before the last one wrote, the digit
histograms, the count, the tickets, before waiting for the last one saw unfinished values in about one view of
three hundred.) Beside them twenty-one scenes of a view each, whose emits are the most CTAs, and one scene's views
that do share their launches."""
import numpy as np
import pytest

import webgs
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes,views", [(3, 7), (1, 21), (21, 1)])
def test_views_side_by_side_repeat_their_single_frames(scenes, views):
    specs = [W.SceneSpec(60_000, 4 + s, 1, 64, 20.0) for s in range(scenes)]
    packed = [s.build() for s in specs]
    cams = [[c.view() for _, c in W.orbit_cameras(views, 17 + s, 9.0, resolutions=((96, 64), (128, 96)))] for s in range(scenes)]
    want = []
    with webgs.Context(flags=webgs.GS_FLAG_NO_GRAPH) as ctx:
        for spec, p, vs in zip(specs, packed, cams):
            sc = ctx.upload(p, spec.count)
            want += [ctx.forward(sc, v)["rgba8"] for v in vs]
            sc.close()
    for _ in range(40):
        with webgs.Context() as ctx:
            scs = [ctx.upload(p, s.count) for p, s in zip(packed, specs)]
            out = ctx.forward_batch([(sc, v) for sc, vs in zip(scs, cams) for v in vs])
            for sc in scs:
                sc.close()
        for a, b in zip(want, out):
            np.testing.assert_array_equal(a, b["rgba8"])
