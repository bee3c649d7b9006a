"""A colour that is not finite under a finite dL/drgb: the running sum of the pixels that blend it stops being
finite, which may reach the Gaussians that those pixels blend and no others. Every Gaussian without a pixel in
common with it keeps the gradient that it has when the colour is finite.

Tolerance: two runs that add the same terms in another order agree to 1e-5 of the largest entry."""
import numpy as np
import pytest

import webgs
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.inf, 3.0e38])
@pytest.mark.parametrize("tile", [8, 16, 32])
def test_a_gaussian_without_a_finite_colour(tile, bad):
    n, w, h = 600, 96, 80
    packed = W.SceneSpec(n, 78, 0).build()
    packed[3 * n:6 * n] -= 0.5  # small splats: a block of pixels meets many that its pixels do not all blend
    packed[:3] = (0.3, 0.2, 3.0)  # behind the others, so that they are visited after it
    dc = packed[10 * n:13 * n].reshape(n, 3)
    view = W.CameraSpec((0.0, 0.0, -4.0), (0, 0, 0), 60.0, w, h).view()
    dl = np.random.default_rng(6).normal(0.0, 30.0 if np.isfinite(bad) else 1e-3, (h, w, 3)).astype(np.float32)
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE, tile_size=tile) as ctx:
        def frame(dl):
            sc = ctx.upload(packed, n)
            rgb = ctx.forward(sc, view, rgba8=False, rgb=True)["rgb"]
            g = ctx.backward(sc, dl)
            sc.close()
            return rgb, g

        dc[0] = (1.0, 1.0, 1.0)
        rgb, want = frame(dl)
        dc[0] = (9.0, 1.0, 1.0)
        pixels = (frame(dl)[0] != rgb).any(2)  # that blend Gaussian 0
        assert 4 < pixels.sum() < w * h // 4
        shared = frame(np.where(pixels[..., None], dl, 0.0).astype(np.float32))[1]
        apart = (shared[10 * n:13 * n].reshape(n, 3) == 0.0).all(1)  # Gaussians with no pixel in common with it
        dc[0] = (bad, 1.0, 1.0)
        got = frame(dl)[1]
    assert apart.sum() > n // 2 and not apart[0]
    at = 0
    for width in (3, 3, 4, 3, 1, 45):
        g, ref = got[at * n:(at + width) * n].reshape(n, width)[apart], want[at * n:(at + width) * n].reshape(n, width)[apart]
        at += width
        assert np.isfinite(g).all(), width
        assert np.abs(g - ref).max() <= 1e-5 * np.abs(ref).max(), width


def test_no_finite_gradient_anywhere_costs_no_multiple_of_a_finite_one():
    """A diverged step (dL/drgb all NaN). Blocks with such a pixel sum their hits by selects and shuffles: 1.0 ms
    against 0.33 of a finite step at 1M / 1080p. Pixels that walk their lists one by one take fifteen times as long,
    so the bound is 6."""
    spec, cam = W.SceneSpec(300_000, 2, 1, 64, 20.0), W.CAMERA_720P
    dl = np.random.default_rng(8).normal(0.0, 1e-3, (cam.height, cam.width, 3)).astype(np.float32)
    ms = []
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE | webgs.GS_FLAG_PROFILE) as ctx:
        sc = ctx.upload(spec.build(), spec.count)
        for d in (dl, np.full_like(dl, np.nan)):
            times = []
            for _ in range(5):
                ctx.forward(sc, cam.view(), rgba8=False, rgb=True)
                ctx.backward(sc, d)
                times.append(ctx.timings()["raster backward"]["ms"])
            ms.append(min(times))
        sc.close()
    print(ms)
    assert ms[1] <= 6.0 * ms[0], ms
